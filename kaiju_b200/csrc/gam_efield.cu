// Constrained-transport electric field (fields.F90:70-232) with shared-memory staging.
//
// For each edge direction eD with transverse pair (dT1, dT2) = (J,K), (K,I), (I,J):
//  1. Vf on the dT1 faces, the volume-weighted Central8 of the half-state velocities (the reference's
//     vol*rho*v/max(rho,dFloor) summands) over max(Central8(vol),TINY) -- one pass, k_mom2face3, for all
//     three directions.
//  2. k_edge_tile: a CTA of 256 threads owns a 32 x TJ x TK tile of eD edges. It stages (TMA tensor copies,
//     or cp.async) the stencil footprints -- along dT2: Vf, the dT1 face areas and the dT1 face field
//     (flux/area, half state for the reconstruction, n state for the limiter); along dT1: the dT2 face
//     areas and field; the 2x2 corner densities -- and evaluates GetCornerV, GetCornerD, GetCornerB (two
//     limited EdgeLRs) and the EMF for its edge from shared memory.
#include "gam_efield_tile.cuh"

namespace gam {

// ------------------------------------------------------------------ Mom2Face (fields.F90:235-285)
// Vf at one face (explicit fused multiply-adds): the Central8 sums along dT1 of volume * velocity over that of the
// volumes (clamped at TINY). A is the accumulation type. Double on the FP64 path, which takes the half state's velocities
// (w0..w2) and applies each weight to its volume once for the four sums. Float on the FP32-flux path, whose w0..w2 are the
// products, formed in double by the predictor and rounded once: a velocity rounded to float carries the same error into
// all eight cells, where the products' errors differ from cell to cell, and after 200 steps of the blast wave the gas was
// up to 15% further from the FP64 run's (L1 of the momentum 5.2e-6 against 4.6e-6 at 128^3). Vf is stored as float.
template <typename A>
__device__ __forceinline__ void mom2face_sum(const A* wV, const A* w0, const A* w1, const A* w2, A& f0, A& f1, A& f2) {
    constexpr bool products = sizeof(A) == 4;
    A sV = A(0), s0 = A(0), s1 = A(0), s2 = A(0);
#pragma unroll
    for (int n = 0; n < 8; ++n) {
        const A c8 = A(wC8(n)), w = products ? c8 : c8 * wV[n];
        sV = products ? fma(w, wV[n], sV) : sV + w;
        s0 = fma(w, w0[n], s0);
        s1 = fma(w, w1[n], s1);
        s2 = fma(w, w2[n], s2);
    }
    const A idV = A(1) / (sV > A(TINY) ? sV : A(TINY));   // one reciprocal for the three quotients
    f0 = s0 * idV; f1 = s1 * idV; f2 = s2 * idV;
}

// All three Mom2Face directions in one launch. out.v[eD]: the three component planes the edges of direction eD read
// (dT1 = J, K, I for eD = I, J, K), written over the region of that direction.
//
// Bound by the L1: 8 cells x 4 values per face and direction. So a thread takes several faces of one line of cells and
// keeps the window in registers: RUN faces along j (or k) read RUN + 7 cells each instead of 8 RUN, and 4 faces along i
// are 12 cells in three 16- or 32-byte rows. The blocks of the three directions over the same SLAB k-planes stand next to
// one another in the grid (blockIdx.y = slab), so the planes cross HBM about once. One face and direction at a time, 96
// loads per cell, took 650 us at 256^3 (450 in single precision); now 484 (251).
template <typename A> struct Vf9 { A* v[3][3]; };
constexpr int M2F_TB = 128, SLAB = 8, M2F_RUN = 8;
// blocks per slab of each direction
struct M2fGrid { int bI, bJ, bK, cI, cJ; };   // and 4-face chunks along i, RUN-face chunks along j

template <typename A>
__global__ void __launch_bounds__(M2F_TB) k_mom2face3(Lay L, const A* __restrict__ vol, const A* __restrict__ v0,
                                                      const A* __restrict__ v1, const A* __restrict__ v2, Vf9<A> out,
                                                      Reg rI, Reg rJ, Reg rK, M2fGrid g) {
    constexpr int RUN = M2F_RUN;
    const int slab = blockIdx.y * SLAB;
    const A* const src[4] = {vol, v0, v1, v2};
    int b = blockIdx.x;
    if (b < g.bI) {   // faces along i: 4 per thread, from a multiple of 4 (is = 4)
        int t = b * M2F_TB + threadIdx.x;
        const int ci = t % g.cI;
        t /= g.cI;
        const int j = rI.j0 + t % rI.nj, k = rI.k0 + slab + t / rI.nj;
        if (t / rI.nj >= SLAB || k >= rI.k0 + rI.nk) return;
        const int i0 = rI.i0 + 4 * ci;
        const long long c = L.at(i0, j, k);
        A w[4][12];
#pragma unroll
        for (int q = 0; q < 4; ++q)
#pragma unroll
            for (int r = 0; r < 12; r += 16 / (int)sizeof(A)) {
                if constexpr (sizeof(A) == 8) {
                    const double2 x = __ldg(reinterpret_cast<const double2*>(src[q] + c - 4 + r));
                    w[q][r] = x.x; w[q][r + 1] = x.y;
                } else {
                    const float4 x = __ldg(reinterpret_cast<const float4*>(src[q] + c - 4 + r));
                    w[q][r] = x.x; w[q][r + 1] = x.y; w[q][r + 2] = x.z; w[q][r + 3] = x.w;
                }
            }
        A f[3][4];
#pragma unroll
        for (int m = 0; m < 4; ++m) mom2face_sum<A>(w[0] + m, w[1] + m, w[2] + m, w[3] + m, f[0][m], f[1][m], f[2][m]);
        const bool whole = i0 + 4 <= rI.i0 + rI.ni;
#pragma unroll
        for (int x = 0; x < 3; ++x) {
            A* o = out.v[2][x] + c;
            if (whole) {
                if constexpr (sizeof(A) == 8) {
                    reinterpret_cast<double2*>(o)[0] = make_double2(f[x][0], f[x][1]);
                    reinterpret_cast<double2*>(o)[1] = make_double2(f[x][2], f[x][3]);
                } else *reinterpret_cast<float4*>(o) = make_float4(f[x][0], f[x][1], f[x][2], f[x][3]);
            } else {
#pragma unroll
                for (int m = 0; m < 4; ++m)
                    if (i0 + m < rI.i0 + rI.ni) o[m] = f[x][m];
            }
        }
        return;
    }
    b -= g.bI;
    // a run of faces along j or k from the face at (i, f0): cells f0 - 4 .. f0 + RUN + 2
    auto run = [&](int first, int last, long long c, long long s, A* const* o) {
        A w[4][RUN + 7];
#pragma unroll
        for (int n = 0; n < RUN + 7; ++n)
            if (n < 8 || first + n - 8 < last)   // the last cell that a face of this run reads
#pragma unroll
                for (int q = 0; q < 4; ++q) w[q][n] = __ldg(src[q] + c + (long long)(n - 4) * s);
#pragma unroll
        for (int m = 0; m < RUN; ++m) {
            if (first + m > last) break;
            A f0, f1, f2;
            mom2face_sum<A>(w[0] + m, w[1] + m, w[2] + m, w[3] + m, f0, f1, f2);
            const long long cm = c + m * s;
            o[0][cm] = f0; o[1][cm] = f1; o[2][cm] = f2;
        }
    };
    if (b < g.bJ) {
        int t = b * M2F_TB + threadIdx.x;
        const int i = rJ.i0 + t % rJ.ni;
        t /= rJ.ni;
        const int j = rJ.j0 + RUN * (t % g.cJ), k = rJ.k0 + slab + t / g.cJ;
        if (t / g.cJ >= SLAB || k >= rJ.k0 + rJ.nk) return;
        run(j, rJ.j0 + rJ.nj - 1, L.at(i, j, k), L.P, out.v[0]);
        return;
    }
    b -= g.bJ;
    {
        const int t = b * M2F_TB + threadIdx.x;
        const int i = rK.i0 + t % rK.ni, j = rK.j0 + t / rK.ni;
        if (j >= rK.j0 + rK.nj) return;
        static_assert(SLAB % RUN == 0, "runs of a slab");
        for (int k = rK.k0 + slab; k < rK.k0 + slab + SLAB && k < rK.k0 + rK.nk; k += RUN)
            run(k, rK.k0 + rK.nk - 1, L.at(i, j, k), (long long)L.P * L.Q, out.v[1]);
    }
}

template <typename A>
static void launch_mom2face(const Lay& L, const A* vol, const A* v0, const A* v1, const A* v2, const Vf9<A>& out,
                            const Reg& rI, const Reg& rJ, const Reg& rK, cudaStream_t st) {
    constexpr int RUN = M2F_RUN;
    M2fGrid g;
    g.cI = (rI.ni + 3) / 4;
    g.cJ = (rJ.nj + RUN - 1) / RUN;
    g.bI = (int)nblk((long long)g.cI * rI.nj * SLAB, M2F_TB);
    g.bJ = (int)nblk((long long)rJ.ni * g.cJ * SLAB, M2F_TB);
    g.bK = (int)nblk((long long)rK.ni * rK.nj, M2F_TB);
    const int nk = rI.nk > rJ.nk ? (rI.nk > rK.nk ? rI.nk : rK.nk) : (rJ.nk > rK.nk ? rJ.nk : rK.nk);
    k_mom2face3<A><<<dim3((unsigned)(g.bI + g.bJ + g.bK), (unsigned)((nk + SLAB - 1) / SLAB)), M2F_TB, 0, st>>>(
        L, vol, v0, v1, v2, out, rI, rJ, rK, g);
}

void efield_kernels_init() {
    set_edge_smem<double, double, 0>(); set_edge_smem<double, double, 1>(); set_edge_smem<double, double, 2>();
    efield_kernels_init_f32();
}

// CalcElecField (fields.F90:70-232): E = 0, then for eD = I, J, K: Mom2Face along dT1, EMF on the edges (the three
// directions beside one another)
void enqueue_efield(Handle& h, const StateP& nS, Branches& br) {
    (void)nS;   // the limiter values come from the precomputed nbA planes
    cudaStream_t st = br.st;
    const Lay& L = h.L;
    // E = 0 (fields.F90:88) needs no pass per step: the edge kernels rewrite the same edges every step, and
    // every edge outside them stays zero from the pool's zeroing (initialisation clears its scratch use)
    GridP g = h.gridP();
    EdgeSrc<double> in64;
    EdgeSrc<float> in32;
    if (h.prec == PREC_FP32FLUX) {
        const F32Planes& f = h.f32;
        for (int x = 0; x < 3; ++x) in32.Vf[x] = f.Vf[x];
        for (int d = 0; d < 3; ++d) {
            in32.face[d] = f.face[d]; in32.hbA[d] = f.hbA[d]; in32.nbA[d] = f.nbA[d]; in32.edge[d] = f.edge[d];
            for (int c = 0; c < 6; ++c) in32.Te[d][c] = f.Te[d][c];
            for (int c = 0; c < 4; ++c) in32.Teb[d][c] = f.Teb[d][c];
            for (int c = 0; c < 2; ++c) in32.edgB0[d][c] = f.edgB0[d][c];
        }
        in32.rho = f.Wh[0];
    } else {
        for (int x = 0; x < 3; ++x) in64.Vf[x] = h.Vf[x];
        for (int d = 0; d < 3; ++d) {
            in64.face[d] = h.face[d]; in64.hbA[d] = h.hbA[d]; in64.nbA[d] = h.nbA[d]; in64.edge[d] = h.edge[d];
            for (int c = 0; c < 6; ++c) in64.Te[d][c] = h.Te[d][3 + c];
            for (int c = 0; c < 4; ++c) in64.Teb[d][c] = h.Teb[d][c];
            for (int c = 0; c < 2; ++c) in64.edgB0[d][c] = h.edgB0[d][c];
        }
        in64.rho = h.Wh[0];
    }
    int is = L.is(), ie = L.ie(), js = L.js(), je = L.je(), ks = L.ks(), ke = L.ke();
    bool f32 = h.prec == PREC_FP32FLUX;
    // Mom2Face regions (dT1 = J, K, I for the I, J, K edges) and the edge regions
    const Reg rv[3] = {mkreg(0, L.Ni - 1, js, je + 1, 0, L.Nk - 1), mkreg(0, L.Ni - 1, 0, L.Nj - 1, ks, ke + 1),
                       mkreg(is, ie + 1, 0, L.Nj - 1, 0, L.Nk - 1)};
    const Reg re[3] = {mkreg(is, ie, js, je + 1, ks, ke + 1), mkreg(is, ie + 1, js, je, ks, ke + 1),
                       mkreg(is, ie + 1, js, je + 1, ks, ke)};
    if (f32) {
        Vf9<float> o;
        for (int x = 0; x < 3; ++x) { o.v[0][x] = h.f32.VfE[0][x]; o.v[1][x] = h.f32.VfE[1][x]; o.v[2][x] = h.f32.Vf[x]; }
        float* const* w = h.f32.VdV;
        launch_mom2face<float>(L, h.f32.volume, w[0], w[1], w[2], o, rv[2], rv[0], rv[1], st);
    } else {
        Vf9<double> o;
        for (int x = 0; x < 3; ++x) { o.v[0][x] = h.VfE[0][x]; o.v[1][x] = h.VfE[1][x]; o.v[2][x] = h.Vf[x]; }
        launch_mom2face<double>(L, g.volume, h.Wh[1], h.Wh[2], h.Wh[3], o, rv[2], rv[0], rv[1], st);
    }
    h.launches++;
    for (int eD = 2; eD >= 0; --eD) {   // the last on the main branch
        if (eD > 0) br.go(SIDE_EDGE + eD - 1);
        for (int x = 0; x < 3; ++x) {
            in32.Vf[x] = eD < 2 ? h.f32.VfE[eD][x] : h.f32.Vf[x];
            in64.Vf[x] = eD < 2 ? h.VfE[eD][x] : h.Vf[x];
        }
        if (f32) launch_edge_dir_f32(h, in32, eD, re[eD], st);
        else launch_edge_dir<double, double>(h, in64, eD, re[eD], st);
        if (eD > 0) br.back();
    }
    br.join(SIDE_EDGE);
    br.join(SIDE_EDGE + 1);
}

}  // namespace gam
