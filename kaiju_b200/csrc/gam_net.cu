// The closure network's kernels: weight packing, the tcgen05 implicit-GEMM convolution (forward and
// backward-data), the weight gradient, the bias gradient and Adam. Layout and GEMM mapping: gam_net.cuh.
#include <cstdio>

#include "gam_net.cuh"
#include "gam_tc.cuh"
#include "gam_tma.cuh"

namespace gam {
namespace {

constexpr uint32_t WAIT_LIMIT = 1u << 24;   // mbarrier polls before a wait gives up (well above any MMA time)

__device__ __forceinline__ float gelu(float x) { return 0.5f * x * (1.0f + erff(x * 0.70710678118654752f)); }
__device__ __forceinline__ float gelu_d(float x) {
    return 0.5f * (1.0f + erff(x * 0.70710678118654752f)) + x * 0.39894228040143268f * expf(-0.5f * x * x);
}
__device__ __forceinline__ uint32_t pack2(float a, float b) {
    __nv_bfloat162 h = __floats2bfloat162_rn(a, b);   // a at the lower address
    return *reinterpret_cast<uint32_t*>(&h);
}

enum { MODE_HIDDEN = 0, MODE_OUT = 1, MODE_BWD = 2 };

struct ConvArgs {
    const __nv_bfloat16* gz;   // MODE_BWD: pre-activation of the previous layer (pitch 32): the epilogue
                               // multiplies the input gradient by its GELU derivative
    const __nv_bfloat16* w;    // packed weights, 27 taps of [32 x CINP] K-major blocks
    const float* bias;         // [cout] (MODE_HIDDEN, MODE_OUT)
    __nv_bfloat16* y;          // MODE_HIDDEN: GELU(z); MODE_BWD: the previous layer's gradient (pitch 32)
    __nv_bfloat16* z;          // MODE_HIDDEN: pre-activation (null: not kept), pitch 32
    float* yf;                 // MODE_OUT: output planes [cout][E]
    long long E, c0, c1;
    int P, Q, cout;
    int* err;
};

constexpr int ROWS = 128;        // cells of a window: the M of a tile
constexpr int TILE = ROWS - 2;   // output cells of a tile (its first and last rows only feed their neighbours)

template <int CINP>
struct ConvShape {
    static constexpr int WIN = ROWS * CINP * 2;        // a window: 128 cells x CINP channels, swizzled rows
    static constexpr int TAPB = 32 * CINP * 2;         // one tap's packed weights
    static constexpr int WB = (27 * TAPB + 1023) / 1024 * 1024;   // all taps, resident for the CTA's life
    static constexpr int NS = CINP == 32 ? 5 : 12;     // window stages in the ring
    // two CTAs per SM, no more: each holds 256 of the SM's 512 TMEM columns
    static constexpr int BYTES = WB + NS * WIN + 1024;
    static constexpr int THREADS = 192;                // 4 epilogue warps, 1 MMA warp, 1 copy warp
    static_assert(2 * (BYTES + 4096) <= 227 * 1024 && 3 * BYTES > 227 * 1024, "two CTAs per SM");
};

__device__ __forceinline__ unsigned char* align1k(unsigned char* p) {
    uint32_t s = tc::smem_u32(p);
    return p + ((1024u - (s & 1023u)) & 1023u);
}

__device__ __forceinline__ void mbar_arrive(uint64_t* mbar) {
    asm volatile("{\n\t.reg .b64 st;\n\tmbarrier.arrive.shared::cta.b64 st, [%0];\n\t}" :: "r"(tc::smem_u32(mbar))
                 : "memory");
}
__device__ __forceinline__ void epi_barrier() { asm volatile("bar.sync 1, 128;" ::: "memory"); }

// out[c][n] = sum over the 27 taps t and input channels k of in[c + off(t)][k] * W_t[n][k].
//
// The three taps di = -1, 0, +1 of a (dj, dk) pair read the same cells, one row apart. One MMA takes all three at
// once, N = 96 output columns: D[r][di * 32 + n] = sum over (dj, dk), k of in[cell(r) + off(dj, dk)][k] * W[n][k], and
// the epilogue adds out[c] = D[c-1][di=-1] + D[c][di=0] + D[c+1][di=+1] (a lane shuffle, and a row each side of a warp
// through shared memory). The A operand is then read from shared memory once instead of three times -- with N = 32
// that read, not the math, set the MMA's time -- and it needs no shifted start, so a window is a plain 128 x CINP box
// that one tensor copy brings in swizzled, with no copy instructions in the other warps. No unit is near
// its limit (32 channels, 64^3: math 21%, L2 27%, issue 45%); the 16- and the 32-channel layers, with half and twice the
// bytes and MMAs, take almost the same time, so what is left goes with the nine windows of a tile, one after the other.
// Warps 0-3: epilogue (warp w reads TMEM lanes 32w..32w+31). One thread of warp 4 issues the MMAs of a window once
// full[s] completes, commits them to empty[s] and, after a tile's last window, to tfull[a]; one thread of warp 5 fills
// the ring of NS windows. Two TMEM accumulators alternate; tempty[a] completes when the epilogue has read one.
// 128^3 (137 x 137 x 144 cells): 32 -> 32 channels 533 -> 291 us, 32 -> 27 514 -> 256, 16 -> 32 317 -> 261, against
// per-thread 16-byte copies, N = 32 and the epilogue in the copying warps.
template <int CINP, int MODE>
__global__ void __launch_bounds__(192, 2) k_conv(const __grid_constant__ CUtensorMap xmap, ConvArgs a) {
    using S = ConvShape<CINP>;
    extern __shared__ unsigned char smraw[];
    unsigned char* sW = align1k(smraw);
    unsigned char* sStage = sW + S::WB;
    __shared__ __align__(8) uint64_t full[S::NS], empty[S::NS], tfull[2], tempty[2], wready;
    __shared__ __align__(16) float edge[2][4][2][32];   // [tile parity][warp]: last row's di=-1, first row's di=+1
    __shared__ uint32_t tmemBase;
    __shared__ int failed;
    __shared__ float sBias[32];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

    if (tid < 32) sBias[tid] = (MODE != MODE_BWD && tid < a.cout) ? a.bias[tid] : 0.f;
    if (tid == 0) {
        for (int q = 0; q < S::NS; ++q) { tc::mbar_init(&full[q], 1); tc::mbar_init(&empty[q], 1); }
        for (int q = 0; q < 2; ++q) { tc::mbar_init(&tfull[q], 1); tc::mbar_init(&tempty[q], 128); }
        tc::mbar_init(&wready, 1);
        failed = 0;
        tma::fence_barrier_init();
    }
    if (warp == 0) tc::tmem_alloc(&tmemBase, 256);
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tbase = tmemBase;

    const long long ntiles = (a.c1 - a.c0 + TILE - 1) / TILE;
    const long long myTiles = ntiles > blockIdx.x ? (ntiles - 1 - blockIdx.x) / gridDim.x + 1 : 0;
    auto firstCell = [&](long long T) { return a.c0 + (blockIdx.x + T * (long long)gridDim.x) * TILE - 1; };

    if (warp < 4) {
        // ---------------- epilogues
        bool ok = true;
        for (long long T = 0; T < myTiles; ++T) {
            const int acc = (int)(T & 1);
            // a warp whose wait gave up still meets the others at the barrier of every tile
            ok = __all_sync(0xffffffffu, ok && tc::mbar_wait(&tfull[acc], (uint32_t)((T >> 1) & 1), WAIT_LIMIT));
            const uint32_t t0 = tbase + ((uint32_t)(warp * 32) << 16) + acc * 128;
            float v[32], d[32];
            if (ok) {
                tc::fence_after_sync();
                tc::tmem_ld32(t0, d);   // di = -1: from the row before
                if (lane == 31)
#pragma unroll
                    for (int q = 0; q < 32; q += 4)
                        *reinterpret_cast<float4*>(&edge[acc][warp][0][q]) = make_float4(d[q], d[q + 1], d[q + 2], d[q + 3]);
#pragma unroll
                for (int q = 0; q < 32; ++q) v[q] = __shfl_up_sync(0xffffffffu, d[q], 1);
                tc::tmem_ld32(t0 + 64, d);   // di = +1: from the row after
                if (lane == 0)
#pragma unroll
                    for (int q = 0; q < 32; q += 4)
                        *reinterpret_cast<float4*>(&edge[acc][warp][1][q]) = make_float4(d[q], d[q + 1], d[q + 2], d[q + 3]);
            }
            epi_barrier();
            if (!ok) continue;
            if (lane == 0 && warp > 0)
#pragma unroll
                for (int q = 0; q < 32; ++q) v[q] = edge[acc][warp - 1][0][q];
#pragma unroll
            for (int q = 0; q < 32; ++q) {
                const float up = __shfl_down_sync(0xffffffffu, d[q], 1);
                v[q] += lane == 31 && warp < 3 ? edge[acc][warp + 1][1][q] : up;
            }
            tc::tmem_ld32(t0 + 32, d);
#pragma unroll
            for (int q = 0; q < 32; ++q) v[q] += d[q];
            tc::fence_before_sync();
            mbar_arrive(&tempty[acc]);
            const long long cell = firstCell(T) + tid;
            if (tid == 0 || tid == ROWS - 1 || cell >= a.c1) continue;
            if (MODE == MODE_OUT) {
#pragma unroll
                for (int co = 0; co < 32; ++co)
                    if (co < a.cout) a.yf[(long long)co * a.E + cell] = v[co] + sBias[co];
                continue;
            }
            uint32_t py[16], pz[16];
            if (MODE == MODE_BWD) {
                const uint4* g4 = reinterpret_cast<const uint4*>(a.gz + cell * NET_PITCH);
                uint32_t gz[16];
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    uint4 u = g4[q];
                    gz[4 * q] = u.x; gz[4 * q + 1] = u.y; gz[4 * q + 2] = u.z; gz[4 * q + 3] = u.w;
                }
#pragma unroll
                for (int q = 0; q < 16; ++q) {
                    __nv_bfloat162 h = *reinterpret_cast<__nv_bfloat162*>(&gz[q]);
                    py[q] = pack2(v[2 * q] * gelu_d(__low2float(h)), v[2 * q + 1] * gelu_d(__high2float(h)));
                }
            } else {
#pragma unroll
                for (int q = 0; q < 16; ++q) {
                    const int c0 = 2 * q, c1 = 2 * q + 1;
                    const float z0 = c0 < a.cout ? v[c0] + sBias[c0] : 0.f;
                    const float z1 = c1 < a.cout ? v[c1] + sBias[c1] : 0.f;
                    pz[q] = pack2(z0, z1);
                    py[q] = pack2(gelu(z0), gelu(z1));
                }
            }
            uint4* y4 = reinterpret_cast<uint4*>(a.y + cell * NET_PITCH);
#pragma unroll
            for (int q = 0; q < 4; ++q) y4[q] = make_uint4(py[4 * q], py[4 * q + 1], py[4 * q + 2], py[4 * q + 3]);
            if (MODE == MODE_HIDDEN && a.z) {
                uint4* z4 = reinterpret_cast<uint4*>(a.z + cell * NET_PITCH);
#pragma unroll
                for (int q = 0; q < 4; ++q) z4[q] = make_uint4(pz[4 * q], pz[4 * q + 1], pz[4 * q + 2], pz[4 * q + 3]);
            }
        }
        if (!ok) failed = 1;
    } else if (tid == 128) {
        // ---------------- MMA issue
        const uint32_t idesc = tc::idesc_bf16_f32(128, 96);
        constexpr uint32_t SBO_W = CINP / 8 * 128;
        constexpr uint32_t SWZ = CINP == 32 ? tc::SWZ_64B : tc::SWZ_32B, SBO_X = 8 * CINP * 2;
        long long issued = 0;   // windows whose MMAs were committed
        bool ok = myTiles == 0 || tc::mbar_wait(&wready, 0u, WAIT_LIMIT);
        for (long long T = 0; T < myTiles && ok; ++T) {
            const int acc = (int)(T & 1);
            if (T >= 2 && !tc::mbar_wait(&tempty[acc], (uint32_t)(((T >> 1) - 1) & 1), WAIT_LIMIT)) { ok = false; break; }
            for (int w = 0; w < 9; ++w) {
                const long long it = T * 9 + w;
                const int st = (int)(it % S::NS);
                if (!tc::mbar_wait(&full[st], (uint32_t)((it / S::NS) & 1), WAIT_LIMIT)) { ok = false; break; }
                tc::fence_after_sync();
                const uint32_t win = tc::smem_u32(sStage + st * S::WIN);
                const uint32_t wt = tc::smem_u32(sW) + 3 * w * S::TAPB;   // the taps di = -1, 0, 1 of (dj, dk), 96 rows
#pragma unroll
                for (int ks = 0; ks < CINP / 16; ++ks) {
                    const uint64_t ad = tc::desc_swz(win + ks * 32, 16, SBO_X, SWZ);
                    const uint64_t bd = tc::desc_kmajor(wt + ks * 256, 128, SBO_W);
                    tc::mma_bf16(tbase + acc * 128, ad, bd, idesc, !(w == 0 && ks == 0));
                }
                tc::mma_commit(&empty[st]);
                if (w == 8) tc::mma_commit(&tfull[acc]);
                ++issued;
            }
        }
        if (!ok) {
            failed = 1;
            // the MMAs already issued read shared memory and write TMEM: wait for the last commit
            if (issued > 0) {
                const long long it = issued - 1;
                tc::mbar_wait(&empty[(int)(it % S::NS)], (uint32_t)((it / S::NS) & 1), WAIT_LIMIT);
            }
        }
    } else if (tid == 160 && myTiles > 0) {
        // ---------------- copies
        tma::arrive_expect_tx(&wready, 27 * S::TAPB);
        tma::load_bulk(sW, a.w, 27 * S::TAPB, &wready);
        bool ok = true;
        long long it = 0;
        for (long long T = 0; T < myTiles && ok; ++T) {
            const long long row0 = firstCell(T);
            for (int w = 0; w < 9; ++w, ++it) {
                const int st = (int)(it % S::NS);
                if (it >= S::NS && !tc::mbar_wait(&empty[st], (uint32_t)((it / S::NS - 1) & 1), WAIT_LIMIT)) { ok = false; break; }
                tma::arrive_expect_tx(&full[st], S::WIN);
                tma::load2(sStage + st * S::WIN, &xmap, 0,
                           (int)(row0 + (long long)a.P * ((w % 3 - 1) + (long long)a.Q * (w / 3 - 1))), &full[st]);
            }
        }
        if (!ok) failed = 1;
        // the copies in flight land before the CTA's shared memory goes, whatever became of the other warps
        tc::mbar_wait(&wready, 0u, WAIT_LIMIT);
        for (long long q = it > S::NS ? it - S::NS : 0; q < it; ++q)
            tc::mbar_wait(&full[(int)(q % S::NS)], (uint32_t)((q / S::NS) & 1), WAIT_LIMIT);
    }
    tc::fence_before_sync();
    __syncthreads();
    if (tid == 0 && failed) atomicExch(a.err, 1);
    if (warp == 0) tc::tmem_free(tbase, 256);
}

// ------------------------------------------------------------------ weight gradient
struct DwArgs {
    float* partial;            // [gridDim.x][NG][128][96]
    long long E, c0, c1;
    int P, Q, cin;
    int* err;
};

template <int CINP>
struct DwShape {
    static constexpr int XWIN = ROWS * CINP * 2;          // a window of the layer's input: 128 cells x CINP
    static constexpr int GWIN = ROWS * 32 * 2;            // a window of the gradient: 128 cells x 32
    static constexpr int G = 128 / CINP;                  // windows (dj, dk) per group of 128 rows
    static constexpr int NG = (9 + G - 1) / G;
    static constexpr int STAGE = 9 * XWIN + 3 * GWIN;
    static constexpr int NS = CINP == 32 ? 2 : 3;
    static constexpr int COLS = NG * 96 <= 256 ? 256 : 512;
    // reading warps: four per group, one for the last, whose ninth window is 32 rows at most; MMA issue; copies
    static constexpr int READERS = (NG - 1) * 128 + 32, THREADS = READERS + 64;
    static_assert((NG - 1) * G == 8 && CINP <= 32, "the last group holds one window");
    // the last group's rows beyond the ninth window read what follows it (their results are not used)
    static constexpr int SLACK = NG * G * XWIN > STAGE ? NG * G * XWIN - STAGE : 0;
    static constexpr int BYTES = NS * STAGE + SLACK + 1024;
    static_assert(STAGE % 1024 == 0 && BYTES <= 226 * 1024 && 2 * BYTES > 227 * 1024, "one CTA per SM");
};

// dW[t][co][ci] = sum over cells c of x[c + off(t)][ci] * dy[c][co]. With c' = c + di the three taps of a (dj, dk)
// pair share x[c' + off(dj, dk)] and shift dy instead, so a tile of 128 cells c' takes 9 windows of x and 3 of dy, and
// one MMA contracts 16 of its cells for 4 (or 8) windows' channels (M = 128) against 3 shifts x 32 output channels
// (N = 96). Both operands are MN-major: the rows that a tensor copy brings in are the contraction index, and nothing is
// transposed or copied by threads. Cells outside [c0, c1) have a zero gradient, so the tiles need no masks.
//
// The tensor core truncates when it adds to an accumulator, so the error grows with the number of MMAs added one after
// the other. The accumulators therefore take a chain of 8 at most, and the reading warps add the chains, rounded to
// nearest, in registers (one row and 96 columns per thread); a CTA writes one partial for all its tiles and a fixed-order
// sum in double follows. Boxes so small that two CTAs per SM, taking 16 cells at a time, would add fewer than 8 MMAs each
// have a tile or two per CTA and few partials to sum: chains of 2 there (launch_dw). Against double sums of the same operands, 32-channel layers, 16^3 / 24^3 /
// 32^3 / 40^3: 0.7 / 1.7 / 1.7 / 1.7e-7 (two CTAs per SM adding all they have: 0.9 / 1.7 / 3.1 / 5.1e-7, one: 1.6 / 3.3 /
// 6.0 / 10e-7). The MMAs wait for the readers: a layer's gradient takes 2 to 3 us longer for it at 32^3.
// Building A with 2-byte loads (one per element and tap) took 153 us per 32-channel layer at 32^3; now about 20.
template <int CINP, int CHAIN>
__global__ void __launch_bounds__(DwShape<CINP>::THREADS, 1) k_conv_dw(const __grid_constant__ CUtensorMap xmap,
                                                    const __grid_constant__ CUtensorMap gmap, DwArgs a) {
    using S = DwShape<CINP>;
    extern __shared__ unsigned char smraw[];
    unsigned char* sbase = align1k(smraw);
    __shared__ __align__(8) uint64_t full[S::NS], empty[S::NS], ready, drained, last;
    __shared__ uint32_t tmemBase;
    __shared__ int failed;
    const int tid = threadIdx.x, warp = tid >> 5;
    if (tid == 0) {
        for (int q = 0; q < S::NS; ++q) { tc::mbar_init(&full[q], 1); tc::mbar_init(&empty[q], 1); }
        tc::mbar_init(&ready, 1);
        tc::mbar_init(&drained, S::READERS / 32);
        tc::mbar_init(&last, 1);
        failed = 0;
        tma::fence_barrier_init();
    }
    if (warp == 0) tc::tmem_alloc(&tmemBase, S::COLS);
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tbase = tmemBase;
    const long long ntiles = (a.c1 - a.c0 + 2 + ROWS - 1) / ROWS;   // c' in [c0 - 1, c1 + 1)
    const long long myTiles = ntiles > blockIdx.x ? (ntiles - 1 - blockIdx.x) / gridDim.x + 1 : 0;
    const long long chains = myTiles * (ROWS / 16 / CHAIN);
    if (tid == S::READERS) {
        // ---------------- MMA issue
        const uint32_t idesc = tc::idesc_bf16_f32_mn(128, 96);
        constexpr uint32_t SWZ = CINP == 32 ? tc::SWZ_64B : tc::SWZ_32B, XROW = CINP * 2;
        bool ok = true;
        long long n = 0;   // chains
        for (long long T = 0; T < myTiles && ok; ++T) {
            const int st = (int)(T % S::NS);
            if (!tc::mbar_wait(&full[st], (uint32_t)((T / S::NS) & 1), WAIT_LIMIT)) { ok = false; break; }
            tc::fence_after_sync();
            const uint32_t xw = tc::smem_u32(sbase + st * S::STAGE), gw = xw + 9 * S::XWIN;
            for (int k0 = 0; k0 < ROWS / 16; k0 += CHAIN, ++n) {
                if (n > 0 && !tc::mbar_wait(&drained, (uint32_t)((n - 1) & 1), WAIT_LIMIT)) { ok = false; break; }
                tc::fence_after_sync();
                for (int ks = k0; ks < k0 + CHAIN; ++ks) {
                    const uint64_t bd = tc::desc_swz(gw + ks * 16 * 64, S::GWIN, 8 * 64, tc::SWZ_64B);
#pragma unroll
                    for (int g = 0; g < S::NG; ++g)
                        tc::mma_bf16(tbase + g * 96,
                                     tc::desc_swz(xw + g * S::G * S::XWIN + ks * 16 * XROW, S::XWIN, 8 * XROW, SWZ), bd,
                                     idesc, ks > k0);
                }
                tc::mma_commit(&ready);
            }
            if (ok) tc::mma_commit(&empty[st]);
        }
        if (!ok) {   // the MMAs issued so far complete before the CTA gives its memory back
            failed = 1;
            tc::mma_commit(&last);
            tc::mbar_wait(&last, 0u, WAIT_LIMIT);
        }
    } else if (tid == S::READERS + 32) {
        // ---------------- copies
        bool ok = true;
        long long T = 0;
        for (; T < myTiles; ++T) {
            const int st = (int)(T % S::NS);
            if (T >= S::NS && !tc::mbar_wait(&empty[st], (uint32_t)((T / S::NS - 1) & 1), WAIT_LIMIT)) { ok = false; break; }
            const long long row0 = a.c0 - 1 + (blockIdx.x + T * (long long)gridDim.x) * ROWS;
            unsigned char* dst = sbase + st * S::STAGE;
            tma::arrive_expect_tx(&full[st], S::STAGE);
            for (int w = 0; w < 9; ++w)
                tma::load2(dst + w * S::XWIN, &xmap, 0,
                           (int)(row0 + (long long)a.P * ((w % 3 - 1) + (long long)a.Q * (w / 3 - 1))), &full[st]);
            for (int di = -1; di <= 1; ++di)
                tma::load2(dst + 9 * S::XWIN + (di + 1) * S::GWIN, &gmap, 0, (int)(row0 - di), &full[st]);
        }
        if (!ok) failed = 1;
        for (long long q = T > S::NS ? T - S::NS : 0; q < T; ++q)
            tc::mbar_wait(&full[(int)(q % S::NS)], (uint32_t)((q / S::NS) & 1), WAIT_LIMIT);
    } else if (tid < S::READERS && myTiles > 0) {
        // ---------------- row tid % 128 of group tid / 128
        const int g = tid / 128, row = tid % 128;
        const uint32_t src = tbase + ((uint32_t)((warp & 3) * 32) << 16) + g * 96;
        float acc[96];
#pragma unroll
        for (int q = 0; q < 96; ++q) acc[q] = 0.f;
        bool ok = true;
        for (long long n = 0; n < chains; ++n) {
            ok = __all_sync(0xffffffffu, tc::mbar_wait(&ready, (uint32_t)(n & 1), WAIT_LIMIT));
            if (!ok) break;
            tc::fence_after_sync();
#pragma unroll
            for (int b = 0; b < 3; ++b) {
                float v[32];
                tc::tmem_ld32(src + b * 32, v);
#pragma unroll
                for (int q = 0; q < 32; ++q) acc[b * 32 + q] += v[q];
            }
            tc::fence_before_sync();
            __syncwarp();
            if ((tid & 31) == 0) mbar_arrive(&drained);
        }
        if (!ok) failed = 1;
        else if (g * S::G + row / CINP < 9 && row % CINP < a.cin) {
            float4* out = reinterpret_cast<float4*>(a.partial + (((long long)blockIdx.x * S::NG + g) * 128 + row) * 96);
#pragma unroll
            for (int q = 0; q < 24; ++q) out[q] = make_float4(acc[4 * q], acc[4 * q + 1], acc[4 * q + 2], acc[4 * q + 3]);
        }
    }
    tc::fence_before_sync();
    __syncthreads();
    if (tid == 0 && failed) atomicExch(a.err, 1);
    if (warp == 0) tc::tmem_free(tbase, S::COLS);
}

// grads W[t][co][ci] of one layer = the fixed-order sum of the CTAs' partials: a block per (window, input channel),
// 96 columns (shift, output channel) by 8 slices of the CTAs
template <int CINP>
__global__ void __launch_bounds__(768) k_dw_reduce(const float* partial, int nblk, float* gW, int cin, int cout) {
    using S = DwShape<CINP>;
    __shared__ double red[8][96];
    const int w = blockIdx.x / cin, ci = blockIdx.x % cin, col = threadIdx.x % 96, sl = threadIdx.x / 96;
    const float* q = partial + ((long long)(w / S::G) * 128 + (w % S::G) * CINP + ci) * 96 + col;
    double s = 0.0;
#pragma unroll 4
    for (int b = sl; b < nblk; b += 8) s += q[(long long)b * S::NG * 128 * 96];
    red[sl][col] = s;
    __syncthreads();
    const int co = col % 32;
    if (sl != 0 || co >= cout) return;
    for (int r = 1; r < 8; ++r) s += red[r][col];
    gW[((long long)(3 * w + col / 32) * cout + co) * cin + ci] = (float)s;
}

// bias gradient: per-block partial sums of the gradient w.r.t. the pre-activation over the cell range, then a
// fixed-order sum. A thread reads 8 channels of a cell at once (one channel after the other over the whole range,
// 2 bytes at a time, took 27 us at 32^3, and the final sum by one thread per channel 19 us; now about 6 and 4). The sums run
// in double: a thread adds several cells.
__global__ void __launch_bounds__(256) k_bias_partial(const __nv_bfloat16* dy, long long c0, long long c1, double* part) {
    __shared__ double red[8][32];
    const int tid = threadIdx.x, q = tid & 3;
    double s[8] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    for (long long c = c0 + blockIdx.x * 64LL + (tid >> 2); c < c1; c += gridDim.x * 64LL) {
        const uint4 u = *reinterpret_cast<const uint4*>(dy + c * NET_PITCH + q * 8);
        const uint32_t r[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const __nv_bfloat162 h = *reinterpret_cast<const __nv_bfloat162*>(&r[e]);
            s[2 * e] += __low2float(h);
            s[2 * e + 1] += __high2float(h);
        }
    }
#pragma unroll
    for (int e = 0; e < 8; ++e) {
        for (int o = 4; o < 32; o <<= 1) s[e] += __shfl_xor_sync(0xffffffffu, s[e], o);
        if ((tid & 31) < 4) red[tid >> 5][q * 8 + e] = s[e];
    }
    __syncthreads();
    if (tid < 32) {
        double t = 0.0;
        for (int w = 0; w < 8; ++w) t += red[w][tid];
        part[blockIdx.x * 32 + tid] = t;
    }
}
__global__ void __launch_bounds__(1024) k_bias_reduce(const double* part, int nblk, int cout, float* gb) {
    __shared__ double red[32][33];
    const int co = threadIdx.x & 31, r = threadIdx.x >> 5;
    double s = 0.0;
    for (int b = r; b < nblk; b += 32) s += part[b * 32 + co];
    red[r][co] = s;
    __syncthreads();
    if (r != 0 || co >= cout) return;
    for (int q = 1; q < 32; ++q) s += red[q][co];
    gb[co] = (float)s;
}

// ------------------------------------------------------------------ packing and Adam
// forward blocks: tap t, row n = output channel, K = input channel; backward-data blocks: tap 26 - t (the mirrored
// offset), row n = input channel, K = output channel. All layers in one launch (blockIdx.y); the padding rows and
// channels are zeroed once, when the blocks are allocated (net_clear_weights), and never written.
struct PackArgs {
    const float* W[NET_LAYERS];
    __nv_bfloat16 *fwd[NET_LAYERS], *bwd[NET_LAYERS];
    int cin[NET_LAYERS], cout[NET_LAYERS];
};
__global__ void k_pack(const __grid_constant__ PackArgs a) {
    const int l = blockIdx.y, cin = a.cin[l], cout = a.cout[l];
    const int id = blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= 27 * cout * cin) return;
    const int fCinP = (cin + 15) / 16 * 16, bCinP = (cout + 15) / 16 * 16;
    const int ci = id % cin, co = (id / cin) % cout, t = id / (cin * cout);
    const __nv_bfloat16 w = __float2bfloat16_rn(a.W[l][id]);
    a.fwd[l][((long long)t * 32 * fCinP * 2 + tc::kmajor_off(co, ci, fCinP)) / 2] = w;
    if (a.bwd[l]) a.bwd[l][((long long)(26 - t) * 32 * bCinP * 2 + tc::kmajor_off(ci, co, bCinP)) / 2] = w;
}

__global__ void k_adam(float* p, const float* g, float* m, float* v, long long n, float lr, float b1, float b2,
                       float eps, float c1, float c2) {
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.f - b1) * gi;
    const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    p[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
}

inline int pad16(int c) { return (c + 15) / 16 * 16; }

template <typename K>
void set_smem(K kern, int bytes) {
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
}

int g_sms = 0;
int sm_count() {
    if (!g_sms) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&g_sms, cudaDevAttrMultiProcessorCount, dev);
        if (g_sms <= 0) g_sms = 148;
    }
    return g_sms;
}

template <int CINP, int MODE>
int launch_conv(const __nv_bfloat16* x, const ConvArgs& a, cudaStream_t st) {
    using S = ConvShape<CINP>;
    CUtensorMap xmap;
    if (!tma::act_map(&xmap, x, CINP, a.E, ROWS)) return (int)cudaErrorInvalidValue;
    const long long ntiles = (a.c1 - a.c0 + TILE - 1) / TILE;
    long long grid = sm_count() * 2;
    if (grid > ntiles) grid = ntiles;
    if (grid < 1) grid = 1;
    k_conv<CINP, MODE><<<(unsigned)grid, S::THREADS, S::BYTES, st>>>(xmap, a);
    return 0;
}

}  // namespace

// shared-memory limits of every kernel instance (set once, outside any stream capture)
int net_init() {
    set_smem(k_conv<16, MODE_HIDDEN>, ConvShape<16>::BYTES);
    set_smem(k_conv<32, MODE_HIDDEN>, ConvShape<32>::BYTES);
    set_smem(k_conv<32, MODE_OUT>, ConvShape<32>::BYTES);
    set_smem(k_conv<32, MODE_BWD>, ConvShape<32>::BYTES);
    set_smem(k_conv_dw<16, 2>, DwShape<16>::BYTES);
    set_smem(k_conv_dw<16, 8>, DwShape<16>::BYTES);
    set_smem(k_conv_dw<32, 2>, DwShape<32>::BYTES);
    set_smem(k_conv_dw<32, 8>, DwShape<32>::BYTES);
    sm_count();
    if (!tma::encoder()) return (int)cudaErrorNotSupported;   // the windows are tensor copies
    return (int)cudaGetLastError();
}

int net_dw_blocks() { return sm_count(); }
long long net_partial_floats(int nblocks) {
    // the largest layer: CINP 32 -> 3 groups of 128 x 96
    return (long long)nblocks * DwShape<32>::NG * 128 * 96;
}
size_t net_act_bytes(long long E) { return (size_t)E * sizeof(__nv_bfloat16); }

int net_clear_weights(__nv_bfloat16* wfwd[NET_LAYERS], __nv_bfloat16* wbwd[NET_LAYERS], cudaStream_t st) {
    NetShape s = net_shape();
    for (int l = 0; l < NET_LAYERS; ++l) {
        cudaMemsetAsync(wfwd[l], 0, sizeof(__nv_bfloat16) * 27 * pad16(s.cin[l]) * 32, st);
        if (wbwd[l]) cudaMemsetAsync(wbwd[l], 0, sizeof(__nv_bfloat16) * 27 * pad16(s.cout[l]) * 32, st);
    }
    return (int)cudaGetLastError();
}

int net_pack_weights(const float* params, __nv_bfloat16* wfwd[NET_LAYERS], __nv_bfloat16* wbwd[NET_LAYERS],
                     cudaStream_t st) {
    NetShape s = net_shape();
    PackArgs a{};
    int most = 0;
    for (int l = 0; l < NET_LAYERS; ++l) {
        a.W[l] = params + net_param_offset(l);
        a.fwd[l] = wfwd[l]; a.bwd[l] = wbwd[l];
        a.cin[l] = s.cin[l]; a.cout[l] = s.cout[l];
        const int n = 27 * s.cin[l] * s.cout[l];
        if (n > most) most = n;
    }
    k_pack<<<dim3((most + 255) / 256, NET_LAYERS), 256, 0, st>>>(a);
    return (int)cudaGetLastError();
}

int net_forward(const NetBox& b, __nv_bfloat16* const wfwd[NET_LAYERS], const float* params, NetBuffers& nb,
                bool keepPre, int* err, cudaStream_t st) {
    NetShape s = net_shape();
    for (int l = 0; l < NET_LAYERS; ++l) {
        ConvArgs a{};
        a.w = wfwd[l];
        a.bias = params + net_param_offset(l) + 27LL * s.cout[l] * s.cin[l];
        a.E = b.E; a.c0 = b.c0; a.c1 = b.c1; a.P = b.P; a.Q = b.Q;
        a.cout = s.cout[l];
        a.err = err;
        int rc;
        if (l < NET_LAYERS - 1) {
            a.y = nb.act[l + 1];
            a.z = keepPre ? nb.pre[l] : nullptr;
            if (l == 0) rc = launch_conv<16, MODE_HIDDEN>(nb.act[l], a, st);
            else rc = launch_conv<32, MODE_HIDDEN>(nb.act[l], a, st);
        } else {
            a.yf = nb.out;
            rc = launch_conv<32, MODE_OUT>(nb.act[l], a, st);
        }
        if (rc) return rc;
    }
    return (int)cudaGetLastError();
}

template <int CINP>
static int launch_dw(const __nv_bfloat16* x, const __nv_bfloat16* dy, const DwArgs& a, int nblk, float* gW, int cout,
                     cudaStream_t st) {
    using S = DwShape<CINP>;
    CUtensorMap xmap, gmap;
    if (!tma::act_map(&xmap, x, CINP, a.E, ROWS) || !tma::act_map(&gmap, dy, NET_PITCH, a.E, ROWS))
        return (int)cudaErrorInvalidValue;
    const long long ntiles = (a.c1 - a.c0 + 2 + ROWS - 1) / ROWS;
    const int grid = ntiles < nblk ? (int)ntiles : nblk;
    const long long spread = ntiles * (ROWS / 16) / (2 * sm_count());   // 16-cell MMAs per CTA, two CTAs per SM
    if (spread >= 8) k_conv_dw<CINP, 8><<<grid, S::THREADS, S::BYTES, st>>>(xmap, gmap, a);
    else k_conv_dw<CINP, 2><<<grid, S::THREADS, S::BYTES, st>>>(xmap, gmap, a);
    k_dw_reduce<CINP><<<9 * a.cin, 768, 0, st>>>(a.partial, grid, gW, a.cin, cout);
    return 0;
}

// gradients of every parameter from the output gradient nb.grad[3] (channels-last, pitch 32), given the
// activations and pre-activations of the last forward (keepPre)
int net_backward(const NetBox& b, __nv_bfloat16* const wbwd[NET_LAYERS], NetBuffers& nb, float* grads, int* err,
                 cudaStream_t st) {
    NetShape s = net_shape();
    const int nblk = net_dw_blocks();
    for (int l = NET_LAYERS - 1; l >= 0; --l) {
        DwArgs d{};
        d.partial = nb.partial;
        d.E = b.E; d.c0 = b.c0; d.c1 = b.c1; d.P = b.P; d.Q = b.Q; d.cin = s.cin[l]; d.err = err;
        float* gW = grads + net_param_offset(l);
        int rc = l == 0 ? launch_dw<16>(nb.act[l], nb.grad[l], d, nblk, gW, s.cout[l], st)
                        : launch_dw<32>(nb.act[l], nb.grad[l], d, nblk, gW, s.cout[l], st);
        if (rc) return rc;
        double* bpart = reinterpret_cast<double*>(nb.partial);   // the weights' partials have been summed
        k_bias_partial<<<nblk, 256, 0, st>>>(nb.grad[l], b.c0, b.c1, bpart);
        k_bias_reduce<<<1, 1024, 0, st>>>(bpart, nblk, s.cout[l], gW + 27LL * s.cout[l] * s.cin[l]);
        if (l > 0) {   // gradient w.r.t. the previous layer's pre-activation: through this layer, then GELU'
            ConvArgs a{};
            a.gz = nb.pre[l - 1]; a.w = wbwd[l];
            a.y = nb.grad[l - 1];
            a.E = b.E; a.c0 = b.c0; a.c1 = b.c1; a.P = b.P; a.Q = b.Q;
            a.cout = s.cin[l]; a.err = err;
            rc = launch_conv<32, MODE_BWD>(nb.grad[l], a, st);
            if (rc) return rc;
        }
    }
    return (int)cudaGetLastError();
}

int net_adam(float* params, const float* grads, float* m, float* v, long long n, float lr, float b1, float b2,
             float eps, int step, cudaStream_t st) {
    const float c1 = 1.f - powf(b1, (float)step), c2 = 1.f - powf(b2, (float)step);
    k_adam<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(params, grads, m, v, n, lr, b1, b2, eps, c1, c2);
    return (int)cudaGetLastError();
}

}  // namespace gam
