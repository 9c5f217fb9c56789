// GAMERA ideal-MHD step on sm_100a: predictor, constrained-transport E field, interface fluxes,
// update, CFL dt and boundary conditions. One stepGamera (src/gamera/gamapp.F90:73-94) is a fixed
// sequence of kernels on one stream; with the time scalars on the device the sequence is captured
// once per buffer parity as a CUDA graph and replayed.
//
// The flux and E-field kernels compute the reconstruction, limiter and kinetic fluxes in the
// arithmetic type T (double for the plain path, float for the FP32-flux path); state, accumulation,
// CT update, C2P with floors and the dt reduction stay FP64 in both.
#include <cstdio>
#include <cmath>
#include <nvtx3/nvToolsExt.h>
#include "gam_common.cuh"
#include "gam_step.cuh"
#include "gam_lfm.cuh"
#include "gam_kern.cuh"

namespace gam {

// ================================================================================ step scalars
// The predictor's time factors (mhdgroup.F90:459) with AdvanceMHD's trap (:26-28), formed by every thread that needs
// them: a launch of their own took as long as a small problem's kernels
struct StepTimes { double pdt, iodt; };
__device__ __forceinline__ StepTimes step_times(const Scal* sc) {
    const double t = sc->time, dt = sc->dt;
    double ot = sc->otime;
    if (fabs(ot - t) < TINY) ot = t - dt;
    return StepTimes{0.5 * dt, 1.0 / (t - ot)};
}

// ================================================================================ predictor
// Predictor magFlux part (mhdgroup.F90:466-488): AB2 on every face element, ghosts included. Also the
// per-face values EdgeLRs divides out at every stencil point (fields.F90:335-336): flux/max(area,TINY)
// for the half state (reconstruction) and for the limiting state.
struct F32FaceOut { float* hbA[3]; float* nbA[3]; };
struct F32CellOut { float* Wh[5]; float* Wn[5]; float* hb[3]; float* nb[3]; float* VdV[3]; };

// Two consecutive face elements per thread with 16-byte loads and stores (E = P*Q*R is a multiple of 8 and
// every plane starts 16-byte aligned), twice the bytes in flight per thread of a one-element loop; the
// arithmetic per element is unchanged.
__global__ void k_predict_faces(long long E, Par p, GridP g, Vec3P mf, Vec3P omf, Vec3P hmf, Vec3P hbA, Vec3P nbA,
                                F32FaceOut o, const Scal* sc) {
    long long l = 2 * (blockIdx.x * (long long)blockDim.x + threadIdx.x);
    if (l >= E) return;
    const StepTimes tm = step_times(sc);
    const double pdt = tm.pdt, iodt = tm.iodt;   // reciprocals where the reference divides repeatedly
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const double2 Q2 = *reinterpret_cast<const double2*>(mf.v[c] + l);
        const double2 oQ2 = *reinterpret_cast<const double2*>(omf.v[c] + l);
        const double2 a2 = *reinterpret_cast<const double2*>(g.face[c] + l);
        double H[2], hb[2], nb[2];
        const double Q[2] = {Q2.x, Q2.y}, oQ[2] = {oQ2.x, oQ2.y}, A[2] = {a2.x, a2.y};
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            double dQ = (Q[e] - oQ[e]) * iodt;
            H[e] = Q[e] + pdt * dQ;
            const double ia = 1.0 / dmax(A[e], TINY);
            // double precision: rounded once, as the fluxes take the face field from it
            hb[e] = o.hbA[0] ? H[e] * ia : H[e] / dmax(A[e], TINY);
            nb[e] = (p.doLFMLim ? Q[e] : H[e]) * ia;
        }
        if (o.hbA[0]) {
            // the half-state flux, for inspection (in double precision it is hbA times the area)
            *reinterpret_cast<double2*>(hmf.v[c] + l) = make_double2(H[0], H[1]);
            *reinterpret_cast<float2*>(o.hbA[c] + l) = make_float2(float(hb[0]), float(hb[1]));
            *reinterpret_cast<float2*>(o.nbA[c] + l) = make_float2(float(nb[0]), float(nb[1]));
        } else {
            *reinterpret_cast<double2*>(hbA.v[c] + l) = make_double2(hb[0], hb[1]);
            *reinterpret_cast<double2*>(nbA.v[c] + l) = make_double2(nb[0], nb[1]);
        }
    }
}

// bFlux2Fld of the half-state face fluxes (Q + pdt (Q - oQ) / odt) of one cell, for the first steps after a state
// came from outside (Scal::bGiven); out of line and before the cell's other loads, so that the usual path keeps its
// registers, and straight-line, so that its 34 loads are in flight together. As a loop over the faces behind those loads
// it took the predictor phase of a 256^3 step from 1.01 to 1.63 ms (0.94 to 1.58 with FP32 fluxes), now to 1.36 (1.29);
// always from the fluxes, with no field to extrapolate, the phase took 1.51 (1.29).
struct V3 { double x, y, z; };
__device__ __noinline__ V3 half_bxyz(const Lay& L, const GridP& g, const StateP& n, const StateP& o, double pdt,
                                     double iodt, long long c) {
    const long long up[3] = {c + 1, c + L.P, c + (long long)L.P * L.Q};
    double q[6], oq[6];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        q[d] = n.mf[d][c]; q[3 + d] = n.mf[d][up[d]];
        oq[d] = o.mf[d][c]; oq[3 + d] = o.mf[d][up[d]];
    }
    const double idV = 1.0 / g.volume[c];
#pragma unroll
    for (int f = 0; f < 6; ++f) q[f] = q[f] + pdt * ((q[f] - oq[f]) * iodt);
    const double Div = q[3] - q[0] + q[4] - q[1] + q[5] - q[2];
    double B[3];
#pragma unroll
    for (int x = 0; x < 3; ++x) {
        double b = 0.0;
#pragma unroll
        for (int d = 0; d < 3; ++d) b += q[3 + d] * g.xfc[d][x][up[d]] - q[d] * g.xfc[d][x][c];
        B[x] = (b - Div * g.xyzcc[x][c]) * idV;
    }
    return V3{B[0], B[1], B[2]};
}

// bFlux2Fld of the half state + PredictCell (mhdgroup.F90:492-518, 529-563) on every cell, plus the
// BlockCon2Prim primitives of the half state and of state n used by the interface reconstruction.
//
// HBM-bound, so what counts is how little it touches. bFlux2Fld is linear in the face fluxes and the half-state
// fluxes are Q + pdt (Q - oQ) / odt, so the half-state field is the same extrapolation of the two states' Bxyz: 6
// values where the fluxes and their moment arms are 16. Mom2Face forms volume times velocity from the volumes and
// the half-state primitives, and the corner densities are the half-state primitive density, so neither is written
// here in double precision (with FP32 fluxes the products are, mom2face_sum says why); the conserved half state is
// written only for the Boris fluxes (gam_gpu_fetch("hgas") rebuilds it from the primitives). 448 B per zone before, about
// 232 now: 256^3 1.08 -> 0.68 ms, 0.92 -> 0.62 with FP32 fluxes (0.55 without the products).
__global__ void k_predict_cells(const __grid_constant__ Lay L, const __grid_constant__ Par p,
                                const __grid_constant__ GridP g, const __grid_constant__ StateP n,
                                const __grid_constant__ StateP o, StateP h, PrimP Wh, PrimP Wn,
                                F32CellOut f, const Scal* sc) {
    Reg r = {0, L.Ni, 0, L.Nj, 0, L.Nk};
    int i, j, k;
    if (!reg_plane(r, i, j, k)) return;
    long long c = L.at(i, j, k);
    const bool f32 = f.Wh[0] != nullptr;
    const StepTimes tm = step_times(sc);
    const double pdt = tm.pdt, iodt = tm.iodt;
    double Q[5], oQ[5], W[5], oW[5], pW[5], pQ[5], B[3] = {0.0, 0.0, 0.0}, nB[3];
    const bool given = sc->bGiven > 0;
    if (p.doMHD && given) {
        const V3 b = half_bxyz(L, g, n, o, pdt, iodt, c);
        B[0] = b.x; B[1] = b.y; B[2] = b.z;
    }
#pragma unroll
    for (int v = 0; v < 5; ++v) { Q[v] = n.gas[v][c]; oQ[v] = o.gas[v][c]; }
#pragma unroll
    for (int x = 0; x < 3; ++x) nB[x] = n.b[x][c];
    if (p.doMHD && !given) {
#pragma unroll
        for (int x = 0; x < 3; ++x) B[x] = nB[x] + pdt * ((nB[x] - o.b[x][c]) * iodt);
    }
    cellC2P(p, oQ, oW);
    cellC2P(p, Q, W);
#pragma unroll
    for (int v = 0; v < 5; ++v) { double dQ = (W[v] - oW[v]) * iodt; pW[v] = W[v] + pdt * dQ; }
    pW[0] = dmax(pW[0], p.dFloor);
    pW[4] = dmax(pW[4], p.pFloor);
    cellP2C(p, pW, pQ);
    // the conserved half state feeds the Boris flux correction
    if (p.doBoris) {
#pragma unroll
        for (int v = 0; v < 5; ++v) h.gas[v][c] = pQ[v];
    }
    double w[5];
    if (f32) {   // FP32-flux path: float copies of every stencil input
        blockC2P(p, pQ, w);
#pragma unroll
        for (int v = 0; v < 5; ++v) f.Wh[v][c] = float(w[v]);
        blockC2P(p, Q, w);
#pragma unroll
        for (int v = 0; v < 5; ++v) f.Wn[v][c] = float(w[v]);
#pragma unroll
        for (int x = 0; x < 3; ++x) { f.hb[x][c] = float(B[x]); f.nb[x][c] = float(nB[x]); }
        const double V = g.volume[c] * (1.0 / dmax(pQ[0], p.dFloor));   // Mom2Face's summands (fields.F90:265-271)
#pragma unroll
        for (int x = 0; x < 3; ++x) f.VdV[x][c] = float(V * pQ[1 + x]);
        return;
    }
#pragma unroll
    for (int x = 0; x < 3; ++x) h.b[x][c] = B[x];
    blockC2P(p, pQ, w);
#pragma unroll
    for (int v = 0; v < 5; ++v) Wh.w[v][c] = w[v];
    blockC2P(p, Q, w);
#pragma unroll
    for (int v = 0; v < 5; ++v) Wn.w[v][c] = w[v];
}
// the conserved half state from its primitives (FP64 without Boris, for inspection)
__global__ void k_half_con(Lay L, Par p, PrimP Wh, StateP h) {
    int i, j, k;
    if (!reg_plane(Reg{0, L.Ni, 0, L.Nj, 0, L.Nk}, i, j, k)) return;
    const long long c = L.at(i, j, k);
    double w[5], U[5];
    for (int v = 0; v < 5; ++v) w[v] = Wh.w[v][c];
    cellP2C(p, w, U);
    for (int v = 0; v < 5; ++v) h.gas[v][c] = U[v];
}
// the half-state fluxes from the face fields (FP64, for inspection)
__global__ void k_half_flux(long long E, GridP g, Vec3P hbA, Vec3P hmf) {
    const long long l = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (l >= E) return;
    for (int d = 0; d < 3; ++d) hmf.v[d][l] = hbA.v[d][l] * dmax(g.face[d][l], TINY);
}
// Scal::bGiven after a state came from outside: `steps`, raised by k_b_check for a state whose Bxyz is not, bit for
// bit, what a step leaves: bFlux2Fld of its fluxes, with the cells across the axis taking their conjugates'
// (RingFlux2FieldFix). A restart's Bxyz is, so it goes on exactly as the run it was taken from. Tiles take the largest of
// theirs (gam_tiles.cu).
__global__ void k_b_given(Scal* sc, int steps) { sc->bGiven = steps; }
// Both states in one pass over the metrics, by a grid that fits the GPU: a state that differs is known by the first cell
// that does, and the threads then stop (one pass per state by a thread per cell took 0.9 ms of a 60 ms push at 256^3 with
// equal fields and 0.8 with different ones, now 0.8, which is the traffic, and nothing).
__device__ __forceinline__ bool b_differs(const Lay& L, const GridP& g, const StateP& s, long long c, long long src) {
    double B[3];
    cellBxyz(L, g, s.mf, src, B);
    bool same = true;
#pragma unroll
    for (int x = 0; x < 3; ++x) same = same && __double_as_longlong(B[x]) == __double_as_longlong(s.b[x][c]);
    return !same;
}
__global__ void k_b_check(const __grid_constant__ Lay L, const __grid_constant__ Par p, const __grid_constant__ GridP g,
                          const __grid_constant__ StateP n, const __grid_constant__ StateP o, bool doN, bool doO, Scal* sc) {
    const unsigned cells = (unsigned)L.Ni * L.Nj;
    volatile int* given = &sc->bGiven;
    for (int k = blockIdx.y; k < L.Nk; k += gridDim.y)
        for (unsigned t = blockIdx.x * blockDim.x + threadIdx.x; t < cells; t += gridDim.x * blockDim.x) {
            if (*given >= (doN ? B_GIVEN_STEPS : 1)) return;
            const int j = t / (unsigned)L.Ni, i = t - j * (unsigned)L.Ni;
            int jp = j, kp = k;
            if (p.doRing && ((p.ringDoS && j < L.js()) || (p.ringDoE && j > L.je())))
                lfmCC(L, p.ringDoS, p.ringDoE, j, k, jp, kp);
            const long long c = L.at(i, j, k), src = L.at(i, jp, kp);
            const bool dn = doN && b_differs(L, g, n, c, src), dq = doO && b_differs(L, g, o, c, src);
            if (dn) atomicMax(&sc->bGiven, B_GIVEN_STEPS);
            else if (dq) atomicMax(&sc->bGiven, 1);
        }
}

// Flux2Deltas (stress.F90:150-196); O is the flux storage type (float on the FP32-flux path), the sums
// run in double
// Flux2Deltas of one active cell: dGasH (5) and dGasM (3). corr: the learned closure's face corrections
// (24 float planes: direction d, variable v at d*8+v; the 5 gas fluxes then the 3 magnetic-stress momentum
// fluxes), added to the face fluxes, or null.
template <typename O>
__device__ __forceinline__ void cellDeltas(const Lay& L, const Par& p, const GridP& g, const FluxOut<O>& FI,
                                           const FluxOut<O>& FJ, const FluxOut<O>& FK, const float* corr,
                                           long long c, double* dh, double* dm) {
    long long cj = c + L.P, ck = c + (long long)L.P * L.Q;
    double idV = 1.0 / g.volume[c];
    auto cr = [&](int d, int v, long long lo, long long hi) {
        if (!corr) return 0.0;
        const float* q = corr + (long long)(d * 8 + v) * L.E;
        return double(q[lo]) - double(q[hi]);
    };
#pragma unroll
    for (int v = 0; v < 5; ++v)
        dh[v] = (double(FI.g[v][c]) - double(FI.g[v][c + 1]) + double(FJ.g[v][c]) - double(FJ.g[v][cj]) +
                 double(FK.g[v][c]) - double(FK.g[v][ck]) +
                 (cr(0, v, c, c + 1) + cr(1, v, c, cj) + cr(2, v, c, ck))) * idV;
    if (p.doMHD) {
#pragma unroll
        for (int x = 0; x < 3; ++x)
            dm[x] = (double(FI.m[x][c]) - double(FI.m[x][c + 1]) + double(FJ.m[x][c]) - double(FJ.m[x][cj]) +
                     double(FK.m[x][c]) - double(FK.m[x][ck]) +
                     (cr(0, 5 + x, c, c + 1) + cr(1, 5 + x, c, cj) + cr(2, 5 + x, c, ck))) * idV;
        if (p.doBackground) {   // background momentum source (stress.F90:185-188)
#pragma unroll
            for (int x = 0; x < 3; ++x) dm[x] = dm[x] + g.dpB0[x][c];
        }
    }
}

// Flux2Deltas (stress.F90:150-196) into the dGasH/dGasM planes; O is the flux storage type (float on the
// FP32-flux path), the sums run in double. With cond set the kernel runs only when the closure's
// positivity check rejected this step (the plain fallback).
template <typename O>
__global__ void k_flux2deltas(Lay L, Par p, GridP g, FluxOut<O> FI, FluxOut<O> FJ, FluxOut<O> FK, PrimP dGH,
                              Vec3P dGM, const float* corr, const Scal* cond) {
    if (cond && !cond->closureReject) return;
    Reg r = {L.is(), L.Nip, L.js(), L.Njp, L.ks(), L.Nkp};
    int i, j, k;
    if (!reg_plane(r, i, j, k)) return;
    long long c = L.at(i, j, k);
    double dh[5], dm[3] = {0.0, 0.0, 0.0};
    cellDeltas<O>(L, p, g, FI, FJ, FK, corr, c, dh, dm);
#pragma unroll
    for (int v = 0; v < 5; ++v) dGH.w[v][c] = dh[v];
    if (p.doMHD) {
#pragma unroll
        for (int x = 0; x < 3; ++x) dGM.v[x][c] = dm[x];
    }
}

// ================================================================================ update
// E2Flux (fields.F90:18-51) on the active faces; every other face element carries State n over
// (the reference updates State in place after copying it to oState).
__global__ void k_e2flux(Lay L, Par p, Vec3P E, StateP nS, StateP oNew, Reg r, const Scal* sc) {
    int i, j, k;
    if (!reg_plane(r, i, j, k)) return;
    long long c = L.at(i, j, k);
    double m0 = nS.mf[0][c], m1 = nS.mf[1][c], m2 = nS.mf[2][c];
    bool act = p.doMHD && i >= L.is() && i <= L.ie() + 1 && j >= L.js() && j <= L.je() + 1 && k >= L.ks() &&
               k <= L.ke() + 1;
    if (act) {
        double dt = sc->dt;
        long long cj = c + L.P, ck = c + (long long)L.P * L.Q;
        const double* Ei = E.v[0]; const double* Ej = E.v[1]; const double* Ek = E.v[2];
        double dfi = Ek[cj] - Ek[c] - Ej[ck] + Ej[c];
        double dfj = Ei[ck] - Ei[c] - Ek[c + 1] + Ek[c];
        double dfk = Ej[c + 1] - Ej[c] - Ei[cj] + Ei[c];
        m0 = m0 - dt * dfi;
        m1 = m1 - dt * dfj;
        m2 = m2 - dt * dfk;
    }
    oNew.mf[0][c] = m0; oNew.mf[1][c] = m1; oNew.mf[2][c] = m2;
}

__global__ void k_bflux2fld(Lay L, GridP g, StateP s, Reg r) {
    int i, j, k;
    if (!reg_plane(r, i, j, k)) return;
    long long c = L.at(i, j, k);
    double B[3];
    cellBxyz(L, g, s.mf, c, B);
    s.b[0][c] = B[0]; s.b[1][c] = B[1]; s.b[2][c] = B[2];
}
__global__ void k_copy_b(Lay L, StateP src, StateP dst) {
    long long l = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (l >= L.E) return;
    dst.b[0][l] = src.b[0][l]; dst.b[1][l] = src.b[1][l]; dst.b[2][l] = src.b[2][l];
}

__device__ __forceinline__ void normVec3(const double* a, double* o) {
    double nA = sqrt(a[0] * a[0] + a[1] * a[1] + a[2] * a[2]);
    if (nA <= TINY) { o[0] = o[1] = o[2] = 0.0; }
    else { o[0] = a[0] / nA; o[1] = a[1] / nA; o[2] = a[2] / nA; }
}
// CellBoris (mhdgroup.F90:337-390), single fluid
__device__ void cellBoris(const Par& p, double* U2, const double* U0, const double* B2, const double* B0,
                          const double* dGH, const double* dGM, double dt) {
    double W2[5];
    cellC2P(p, U2, W2);
    double D2 = dmax(W2[0], p.dFloor), P2 = dmax(W2[4], p.pFloor);
    double D0 = dmax(U0[0], p.dFloor);
    double V0[3] = {U0[1] / D0, U0[2] / D0, U0[3] / D0};
    double B1[3] = {0.5 * (B2[0] + B0[0]), 0.5 * (B2[1] + B0[1]), 0.5 * (B2[2] + B0[2])};
    double Ca = p.Ca;
    double alpha = (B1[0] * B1[0] + B1[1] * B1[1] + B1[2] * B1[2]) / (D2 * Ca * Ca);
    double dRho = dt * dGH[0];
    double dPGas[3], dPMag[3], dMom[3];
    for (int c = 0; c < 3; ++c) { dPGas[c] = dt * dGH[1 + c]; dPMag[c] = dt * dGM[c]; }
    double pCon = 1.0 / (1.0 + alpha);
    double bh[3];
    normVec3(B1, bh);
    if (alpha > TINY) {
        double s[3] = {dPGas[0] + dPMag[0], dPGas[1] + dPMag[1], dPGas[2] + dPMag[2]};
        double pg = dPGas[0] * bh[0] + dPGas[1] * bh[1] + dPGas[2] * bh[2];
        double ps = s[0] * bh[0] + s[1] * bh[1] + s[2] * bh[2];
        double pv = V0[0] * bh[0] + V0[1] * bh[1] + V0[2] * bh[2];
        for (int c = 0; c < 3; ++c) {
            double para = pg * bh[c];
            double perpS = s[c] - ps * bh[c];
            double perpV = V0[c] - pv * bh[c];
            dMom[c] = (para + pCon * perpS) + alpha * pCon * dRho * perpV;
        }
    } else {
        for (int c = 0; c < 3; ++c) dMom[c] = dPGas[c] + dPMag[c];
    }
    double Wn[5] = {D2, (D0 * V0[0] + dMom[0]) / D2, (D0 * V0[1] + dMom[1]) / D2, (D0 * V0[2] + dMom[2]) / D2, P2};
    cellP2C(p, Wn, U2);
}

// CellReynolds + CellMaxwell/CellBoris (mhdgroup.F90:113-126, 170-197, 263-330) on active cells;
// ghost cells carry State n over.
// FUSED: the deltas are computed here from the face fluxes (Flux2Deltas of the same cell, same arithmetic)
// instead of read from the dGasH/dGasM planes
template <typename O, bool FUSED>
__global__ void k_update_gas(Lay L, Par p, GridP g, StateP nS, StateP oNew, PrimP dGH, Vec3P dGM, FluxOut<O> FI,
                             FluxOut<O> FJ, FluxOut<O> FK, Reg r, const Scal* sc) {
    int i, j, k;
    if (!reg_plane(r, i, j, k)) return;
    long long c = L.at(i, j, k);
    double U[5];
#pragma unroll
    for (int v = 0; v < 5; ++v) U[v] = nS.gas[v][c];
    bool act = i >= L.is() && i <= L.ie() && j >= L.js() && j <= L.je() && k >= L.ks() && k <= L.ke();
    if (act) {
        double dt = sc->dt;
        double dh[5], dm[3] = {0.0, 0.0, 0.0};
        if (FUSED) cellDeltas<O>(L, p, g, FI, FJ, FK, nullptr, c, dh, dm);
        else {
#pragma unroll
            for (int v = 0; v < 5; ++v) dh[v] = dGH.w[v][c];
            if (p.doMHD) { dm[0] = dGM.v[0][c]; dm[1] = dGM.v[1][c]; dm[2] = dGM.v[2][c]; }
        }
        double U0[5];
#pragma unroll
        for (int v = 0; v < 5; ++v) { U0[v] = U[v]; U[v] = U[v] + dt * dh[v]; }
        if (p.doMHD) {
            double dPm[3] = {dm[0], dm[1], dm[2]};
            if (p.doBoris) {
                double B2[3] = {oNew.b[0][c], oNew.b[1][c], oNew.b[2][c]};
                double B0[3] = {nS.b[0][c], nS.b[1][c], nS.b[2][c]};
                if (p.doBackground) {   // total fields (mhdgroup.F90:180-183)
#pragma unroll
                    for (int x = 0; x < 3; ++x) { B2[x] = B2[x] + g.B0[x][c]; B0[x] = B0[x] + g.B0[x][c]; }
                }
                cellBoris(p, U, U0, B2, B0, dh, dPm, dt);
            } else {
                double D = dmax(U[0], p.dFloor), Mx = U[1], My = U[2], Mz = U[3], TotE = U[4];
                const double iD = 1.0 / D;
                double KinE = 0.5 * (sq(Mx) + sq(My) + sq(Mz)) * iD;
                double P = dmax((p.gamma - 1) * (TotE - KinE), p.pFloor);
                Mx = Mx + dt * dPm[0];
                My = My + dt * dPm[1];
                Mz = Mz + dt * dPm[2];
                KinE = 0.5 * (sq(Mx) + sq(My) + sq(Mz)) * iD;
                U[0] = D; U[1] = Mx; U[2] = My; U[3] = Mz; U[4] = KinE + P / (p.gamma - 1);
            }
        }
    }
#pragma unroll
    for (int v = 0; v < 5; ++v) oNew.gas[v][c] = U[v];
}

// bFlux2Fld after EnforceBCs restricted to ghost cells: outside 2.5D the BCs only rewrite faces of
// ghost cells (outer I/J/K faces from ie+2/je+2/ke+2 on, inner ones below is/js/ks), so active cells
// keep the B of the update.
// The ghost cells are enumerated as five slabs so the launch covers only them: k below and above the active
// range (all i, j), then j below and above (all i, active k), then the i ghosts of the active rows (both
// ends of a row next to each other, so a warp reads whole ghost runs of neighbouring rows). i runs fastest
// in every slab.
__host__ __device__ inline long long ghost_cells(const Lay& L) {
    return (long long)L.Ni * L.Nj * L.Nk - (long long)L.Nip * L.Njp * L.Nkp;
}
__device__ __forceinline__ void ghost_ijk(const Lay& L, long long t, int& i, int& j, int& k) {
    const long long sK = (long long)L.Ni * L.Nj, sJ = (long long)L.Ni * L.Nkp;
    const long long nK = sK * (L.Nk - L.Nkp), nJ = sJ * (L.Nj - L.Njp);
    if (t < nK) {   // k slabs: whole (i, j) planes
        const int kk = (int)(t / sK), rem = (int)(t % sK);
        k = kk < L.ks() ? kk : L.ke() + 1 + (kk - L.ks());
        j = rem / L.Ni; i = rem % L.Ni;
        return;
    }
    t -= nK;
    if (t < nJ) {   // j slabs within the active k: whole rows
        const int jj = (int)(t / sJ), rem = (int)(t % sJ);
        j = jj < L.js() ? jj : L.je() + 1 + (jj - L.js());
        k = L.ks() + rem / L.Ni; i = rem % L.Ni;
        return;
    }
    t -= nJ;        // the i ghosts of the active rows: nGi = Ni - Nip cells per row
    const int nGi = L.Ni - L.Nip, ii = (int)(t % nGi), q = (int)(t / nGi);
    i = ii < L.is() ? ii : L.ie() + 1 + (ii - L.is());
    j = L.js() + q % L.Njp; k = L.ks() + q / L.Njp;
}
__global__ void k_bflux2fld_ghost(Lay L, GridP g, StateP s) {
    const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (t >= ghost_cells(L)) return;
    int i, j, k;
    ghost_ijk(L, t, i, j, k);
    long long c = L.at(i, j, k);
    double B[3];
    cellBxyz(L, g, s.mf, c, B);
    s.b[0][c] = B[0]; s.b[1][c] = B[1]; s.b[2][c] = B[2];
}

// ================================================================================ timestep
// CellDT (gridutils.F90:49-106) over the dt domain (one ghost layer at physical boundaries), min-reduced
// The dt domain: one ghost layer at physical boundaries (init.F90:531-537), the active cells with dtActive;
// a tile face has no ghost layer in it (ksDT = ks, keDT = ke; gamapp_mpi.F90:441-462)
__host__ __device__ inline Reg reg_dt(const Lay& L, const Par& p) {
    Reg r = {L.is() - 1, L.Nip + 2, L.js() - 1, L.Njp + 2, L.ks() - 1, L.Nkp + 2};
    if (p.dtActive) r = Reg{L.is(), L.Nip, L.js(), L.Njp, L.ks(), L.Nkp};
    if (!p.dtActive && p.bc[4] == BC_HALO) { r.k0 += 1; r.nk -= 1; }
    if (!p.dtActive && p.bc[5] == BC_HALO) r.nk -= 1;
    return r;
}

// UpdateStateData time bookkeeping (gamapp.F90:113-114, mhdgroup.F90:104-105) and the rest of CalcDT
// (step.F90:103-166): checks, the tFin clamp and the 10*dt0 clamp. mode 1 = initial dt (Hatch). It leaves the next
// step's minimum, NaN count and closure flag cleared.
__device__ __noinline__ void dt_finalize(const Par& p, Scal* sc, int mode) {
    const unsigned long long bits = __ldcg(&sc->dtMinBits);
    const unsigned nan = __ldcg(&sc->nanCount);
    sc->dtMinBits = 0x7FF0000000000000ull;
    sc->nanCount = 0u;
    sc->closureReject = 0;
    if (mode == 0) {
        sc->otime = sc->time;
        sc->time = sc->time + sc->dt;
        sc->ts = sc->ts + 1;
        sc->t = sc->t + sc->dt;
        if (sc->bGiven > 0) sc->bGiven--;
    }
    if (p.fixedTimestep) { sc->status = 0; return; }
    double dtOld = sc->dt;
    double dtMin = __longlong_as_double((long long)bits);
    if (bits >= 0x7FF0000000000000ull || dtMin > HUGEV) dtMin = HUGEV;
    int st = 0;
    if (dtMin == HUGEV) st |= 1;
    if (sc->ts > 0) {
        if (dtOld / dtMin >= 10) st |= 2;
        if ((sc->dt0 > TINY) && (dtMin / sc->dt0 <= p.limDT0)) st |= 2;
        if (dtMin <= TINY) st |= 1;
    }
    if (nan) st |= 4;
    if (sc->waitFail) st |= 8;
    double r = dtMin;
    if ((sc->t + r) > p.tFin) r = dmax(p.tFin - sc->t, TINY);
    if (sc->dt0 > TINY && r > 10.0 * sc->dt0) r = 10.0 * sc->dt0;
    sc->dt = r;
    sc->status = st;
    sc->sticky |= st;
    sc->lastNan = nan;
    sc->waitFail = 0u;   // reported in this step's status (and the sticky OR); the next step starts clear
}
__global__ void k_dt_finalize(const __grid_constant__ Par p, Scal* sc, int mode) { dt_finalize(p, sc, mode); }

// the cells' CFL lengths, fixed with the grid: one plane for CalcDT to read instead of three
__global__ void k_min_length(long long E, const double* di, const double* dj, const double* dk, double* dl) {
    const long long l = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (l >= E) return;
    double m = di[l];
    if (dj[l] < m) m = dj[l];
    if (dk[l] < m) m = dk[l];
    dl[l] = m;
}
// The minimum over the dt domain. finalize >= 0: the last block to finish goes on to finalize the dt in that mode
// (one launch less on the step's chain); -1 where a tiled run reduces the minimum over its tiles first.
__global__ void k_calcdt(Lay L, const __grid_constant__ Par p, GridP g, StateP s, Scal* sc, int finalize) {
    const Reg r = reg_dt(L, p);
    int i, j, k;
    double dtijk = HUGEV * 2.0;
    bool isnan_ = false;
    if (reg_plane(r, i, j, k)) {
        long long c = L.at(i, j, k);
        double rho = s.gas[0][c], ir = 1.0 / rho;   // one reciprocal for the reference's divisions by rho
        double Vx = s.gas[1][c] * ir, Vy = s.gas[2][c] * ir, Vz = s.gas[3][c] * ir;
        double MagV = sqrt(sq(Vx) + sq(Vy) + sq(Vz));
        double ke = 0.5 * rho * sq(MagV);
        double e = s.gas[4][c] - ke;
        double P = (p.gamma - 1) * e;
        double Cs = sqrt(p.gamma * P * ir);
        double Valf = 0.0;
        if (p.doMHD) {
            double Bx = s.b[0][c], By = s.b[1][c], Bz = s.b[2][c];
            if (p.doBackground) { Bx = Bx + g.B0[0][c]; By = By + g.B0[1][c]; Bz = Bz + g.B0[2][c]; }  // gridutils.F90:82-86
            double MagB = sqrt(sq(Bx) + sq(By) + sq(Bz));
            Valf = MagB * rsq(rho);
            if (p.doBoris) Valf = p.Ca * Valf * rsq(p.Ca * p.Ca + Valf * Valf);
        }
        double vCFL = MagV + sqrt(sq(Cs) + sq(Valf)) + 0.0;
        dtijk = p.CFL * g.dl[c] / vCFL;
        if (dtijk != dtijk) { isnan_ = true; dtijk = HUGEV * 2.0; }
    }
    // bit patterns of non-negative doubles order like the values
    unsigned long long bits = __double_as_longlong(dtijk);
    if (dtijk < 0.0) bits = 0ull;
    for (int off = 16; off > 0; off >>= 1) {
        unsigned long long o = __shfl_down_sync(0xffffffffu, bits, off);
        bits = o < bits ? o : bits;
    }
    unsigned nn = __popc(__ballot_sync(0xffffffffu, isnan_));
    __shared__ unsigned long long wmin[32];
    __shared__ unsigned wnan[32];
    int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (lane == 0) { wmin[w] = bits; wnan[w] = nn; }
    __syncthreads();
    if (w == 0) {
        int nw = blockDim.x >> 5;
        bits = lane < nw ? wmin[lane] : ~0ull;
        nn = lane < nw ? wnan[lane] : 0u;
        for (int off = 16; off > 0; off >>= 1) {
            unsigned long long o = __shfl_down_sync(0xffffffffu, bits, off);
            bits = o < bits ? o : bits;
            nn += __shfl_down_sync(0xffffffffu, nn, off);
        }
        if (lane == 0) {
            atomicMin(&sc->dtMinBits, bits);
            if (nn) atomicAdd(&sc->nanCount, nn);
            if (finalize >= 0) {
                __threadfence();
                if (atomicAdd(&sc->blocksDone, 1u) + 1u == gridDim.x * gridDim.y) {
                    __threadfence();
                    sc->blocksDone = 0u;
                    dt_finalize(p, sc, finalize);
                }
            }
        }
    }
}

// ================================================================================ boundary conditions
// EnforceBCs fills I, then J (which also covers the I ghosts), then K, one kernel each. A ghost layer depends on
// active cells only, so every (layer, side) pair is its own row of blocks, and a thread issues all of its loads
// before its first store: the kernels are a few hundred thousand dependent-free copies, bound by the latency of one
// load. One thread per column that walked both sides' four layers, each value loaded after the store before it
// (the planes may alias for the compiler), chained up to 88 load latencies: I / J / K 16.7 / 48 / 46 us at 96x83x70
// periodic and 15.9 / 46 / 27 us at 32x32x4, where the kernels before them take 85 us in all; now
// 6.1 / 4.1 / 4.3 and 4.1 / 3.8 / 3.5 us. At 256^3 with zero gradients 93 / 11 / 10 us, 95 / 15 / 14 before.
//
// Periodic sources are written modulo the extent, which is where the layer-by-layer copies of an extent smaller than
// nG ended up (layer n takes from layer n - extent). withB = 0 inside a step: the bFlux2Fld of the ghost cells that
// follows rewrites every ghost B, so copying it would be dead work; set-up keeps the copied B, as Hatch leaves it.
__device__ __forceinline__ void cpcell(const StateP& s, long long dst, long long src, bool withB) {
    double v[8];
#pragma unroll
    for (int q = 0; q < 5; ++q) v[q] = s.gas[q][src];
    if (withB) { v[5] = s.b[0][src]; v[6] = s.b[1][src]; v[7] = s.b[2][src]; }
#pragma unroll
    for (int q = 0; q < 5; ++q) s.gas[q][dst] = v[q];
    if (withB) { s.b[0][dst] = v[5]; s.b[1][dst] = v[6]; s.b[2][dst] = v[7]; }
}
// the ghost cell dst from src (cell) and the three face fluxes dst[d] from src[d], every load before the first store
__device__ __forceinline__ void cpghost(const StateP& s, bool cell, bool withB, long long cd, long long cs,
                                        const long long* fd, const long long* fs) {
    double v[8], f[3];
    if (cell) {
#pragma unroll
        for (int q = 0; q < 5; ++q) v[q] = s.gas[q][cs];
        if (withB) { v[5] = s.b[0][cs]; v[6] = s.b[1][cs]; v[7] = s.b[2][cs]; }
    }
#pragma unroll
    for (int d = 0; d < 3; ++d) f[d] = s.mf[d][fs[d]];
    if (cell) {
#pragma unroll
        for (int q = 0; q < 5; ++q) s.gas[q][cd] = v[q];
        if (withB) { s.b[0][cd] = v[5]; s.b[1][cd] = v[6]; s.b[2][cd] = v[7]; }
    }
#pragma unroll
    for (int d = 0; d < 3; ++d) s.mf[d][fd[d]] = f[d];
}

// I faces: periodic (bcs.F90:279-327) or zero gradient (bcs.F90:799-843); blockIdx.y = side (0 inner, 1 outer)
__global__ void k_bc_i(Lay L, Par p, GridP g, StateP s, int withB) {
    // one thread per ghost layer n and (j, k) row
    long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    const int nG = L.nG, nj = L.Nj + 1;
    if (t >= (long long)nG * nj * (L.Nk + 1)) return;
    const int n = 1 + (int)(t % nG);
    const long long row = t / nG;
    const int j = (int)(row % nj), k = (int)(row / nj);
    const bool cell = (j < L.Nj) && (k < L.Nk), inner = blockIdx.y == 0;
    const int is = L.is(), ie = L.ie(), bc = p.bc[inner ? 0 : 1];
    if (bc == BC_LFMBW) {
        // the LFM blast wave's fixed shells (ICs/lfmbw.F90:141-225): fixed gas; ghost face fluxes are the
        // conjugate active-shell fluxes scaled by the face areas (J/K signs flip across the axis)
        double dApm[3] = {1.0, 1.0, 1.0};
        if (p.ringDoS && j < L.js()) dApm[1] = dApm[2] = -1.0;
        if (p.ringDoE && j >= L.je() + 1) dApm[1] = dApm[2] = -1.0;
        int ig = inner ? is - n : ie + n;
        double f[3];
        long long cg[3];
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            int di = (!inner && d == 0) ? 1 : 0;
            int ia = inner ? is : ie + di;
            int jp, kp;
            lfmFC(L, p.ringDoS, p.ringDoE, d, j, k, jp, kp);
            cg[d] = L.at(ig + di, j, k);
            long long ca = L.at(ia, jp, kp);
            double dA = g.face[d][cg[d]] / g.face[d][ca];
            f[d] = dApm[d] * dA * s.mf[d][ca];
        }
        if (cell) {
            long long c = L.at(ig, j, k);
            s.gas[0][c] = p.bwD0; s.gas[1][c] = 0.0; s.gas[2][c] = 0.0; s.gas[3][c] = 0.0;
            s.gas[4][c] = p.bwP0 / (p.gamma - 1.0);
        }
#pragma unroll
        for (int d = 0; d < 3; ++d) s.mf[d][cg[d]] = f[d];
    } else if (bc == BC_PERIODIC) {
        const int m = (n - 1) % L.Nip;
        if (inner) {
            long long d = L.at(is - n, j, k), q = L.at(ie - m, j, k);
            const long long fd[3] = {d, d, d}, fs[3] = {q, q, q};
            cpghost(s, cell, withB, d, q, fd, fs);
        } else {
            long long d = L.at(ie + n, j, k), q = L.at(is + m, j, k);
            const long long fd[3] = {d + 1, d, d}, fs[3] = {q + 1, q, q};
            cpghost(s, cell, withB, d, q, fd, fs);
        }
    } else if (bc == BC_ION || bc == BC_WIND) {
        // launch_msph_bcs
    } else if (cell && inner) {
        long long d = L.at(is - n, j, k), q = L.at(is, j, k);
        const long long fd[3] = {d, d, d}, fs[3] = {q, q, q};
        cpghost(s, true, false, d, q, fd, fs);
    } else if (cell) {
        double B[3];
        cellBxyz(L, g, s.mf, L.at(ie, j, k), B);
        long long d = L.at(ie + n, j, k), dI = d + 1;
        double f0 = g.face[0][dI] * (B[0] * g.Tf[0][0][dI] + B[1] * g.Tf[0][1][dI] + B[2] * g.Tf[0][2][dI]);
        double f1 = g.face[1][d] * (B[0] * g.Tf[1][0][d] + B[1] * g.Tf[1][1][d] + B[2] * g.Tf[1][2][d]);
        double f2 = g.face[2][d] * (B[0] * g.Tf[2][0][d] + B[1] * g.Tf[2][1][d] + B[2] * g.Tf[2][2][d]);
        cpcell(s, d, L.at(ie, j, k), false);
        s.mf[0][dI] = f0;
        s.mf[1][d] = f1;
        s.mf[2][d] = f2;
    }
}

// J faces: periodic (bcs.F90:329-378), zero gradient (bcs.F90:845-888) or across the LFM axis (lfmIn / lfmOut,
// bcs.F90:1020-1106: ghosts from their conjugates). blockIdx.y = 2 (n - 1) + side; serial (an axis with fewer than
// nG active rows, whose conjugates reach the other side's ghosts) walks the layers in order in one thread.
__global__ void k_bc_j(Lay L, Par p, StateP s, int withB, int serial) {
    long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    int ni = L.Ni + 1;
    if (t >= (long long)ni * (L.Nk + 1)) return;
    const int i = (int)(t % ni), k = (int)(t / ni);
    const bool cell = (i < L.Ni) && (k < L.Nk);
    const int js = L.js(), je = L.je();
    auto layer = [&](bool inner, int n) {
        const int bc = p.bc[inner ? 2 : 3];
        if (bc == BC_LFMPOLE) {
            const int jg = inner ? js - n : je + n;
            int jp, kp;
            lfmCC(L, p.ringDoS, p.ringDoE, jg, k, jp, kp);
            const long long cs = L.at(i, jp, kp);
            lfmFC(L, p.ringDoS, p.ringDoE, 0, jg, k, jp, kp);
            const double f0 = s.mf[0][L.at(i, jp, kp)];
            const int jf = inner ? jg : jg + 1;   // the first outer J ghost face is je+2
            lfmFC(L, p.ringDoS, p.ringDoE, 1, jf, k, jp, kp);
            const double f1 = -s.mf[1][L.at(i, jp, kp)];
            lfmFC(L, p.ringDoS, p.ringDoE, 2, jg, k, jp, kp);
            const double f2 = -s.mf[2][L.at(i, jp, kp)];
            if (cell) cpcell(s, L.at(i, jg, k), cs, withB);
            s.mf[0][L.at(i, jg, k)] = f0;
            s.mf[1][L.at(i, jf, k)] = f1;
            s.mf[2][L.at(i, jg, k)] = f2;
        } else if (bc == BC_PERIODIC) {
            const int m = (n - 1) % L.Njp;
            if (inner) {
                const long long d = L.at(i, js - n, k), q = L.at(i, je - m, k);
                const long long fd[3] = {d, d, d}, fs[3] = {q, q, q};
                cpghost(s, cell, withB, d, q, fd, fs);
            } else {
                const long long d = L.at(i, je + n, k), q = L.at(i, js + m, k);
                const long long fd[3] = {d, d + L.P, d}, fs[3] = {q, q + L.P, q};
                cpghost(s, cell, withB, d, q, fd, fs);
            }
        } else if (cell) {
            const long long d = L.at(i, inner ? js - n : je + n, k), q = L.at(i, inner ? js : je, k);
            const long long up = inner ? 0 : L.P;   // the outer J faces je+2.. repeat face je+1
            const long long fd[3] = {d, d + up, d}, fs[3] = {q, q + up, q};
            cpghost(s, true, false, d, q, fd, fs);
        }
    };
    if (!serial) { layer((blockIdx.y & 1) == 0, 1 + (int)(blockIdx.y >> 1)); return; }
    for (int side = 0; side < 2; ++side)
        for (int n = 1; n <= L.nG; ++n) layer(side == 0, n);
}

// K faces: periodic (bcs.F90:380-450, 2.5D replication included) or zero gradient (bcs.F90:890-930); a tile's halo
// faces are filled from the neighbouring tile after the step. blockIdx.y = 2 (n - 1) + side
__global__ void k_bc_k(Lay L, Par p, StateP s, int withB) {
    long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    int ni = L.Ni + 1;
    if (t >= (long long)ni * (L.Nj + 1)) return;
    const int i = (int)(t % ni), j = (int)(t / ni);
    const bool cell = (i < L.Ni) && (j < L.Nj), inner = (blockIdx.y & 1) == 0;
    const int ks = L.ks(), ke = L.ke(), n = 1 + (int)(blockIdx.y >> 1), bc = p.bc[inner ? 4 : 5];
    const long long PQ = (long long)L.P * L.Q;
    if (bc == BC_HALO) return;
    if (bc == BC_PERIODIC) {
        const int m = (n - 1) % L.Nkp;
        if (inner || p.do25D) {
            const long long d = L.at(i, j, inner ? ks - n : ks + n), q = L.at(i, j, p.do25D ? ks : ke - m);
            const long long fd[3] = {d, d, d}, fs[3] = {q, q, q};
            cpghost(s, cell, withB, d, q, fd, fs);
        } else {
            const long long d = L.at(i, j, ke + n), q = L.at(i, j, ks + m);
            const long long fd[3] = {d, d, d + PQ}, fs[3] = {q, q, q + PQ};
            cpghost(s, cell, withB, d, q, fd, fs);
        }
    } else if (cell && inner) {
        const long long d = L.at(i, j, ks - n), q = L.at(i, j, ks);
        const long long fd[3] = {d, d, d}, fs[3] = {q, q, q};
        cpghost(s, true, false, d, q, fd, fs);
    } else if (cell) {
        const long long d = L.at(i, j, ke + n), q = L.at(i, j, ke);
        // bcs.F90:924 writes the J component of face ke+1 into the K faces above it; kept for parity. That face is
        // the first ghost layer's, by then a copy of the J face of ke.
        const double f0 = s.mf[0][q], f1 = s.mf[1][q];
        cpcell(s, d, q, false);
        s.mf[0][d] = f0;
        s.mf[1][d] = f1;
        s.mf[2][d + PQ] = f1;
    }
}

// All six sides periodic: EnforceBCs and the bFlux2Fld of the ghost cells in one launch. The three sweeps copy along one
// axis each, so a ghost value is that of the active element its three indices map to one by one (images of other
// images never arise, and what is read is never written); the field of a ghost cell comes from the fluxes its six faces
// get. The update then need not carry over more than the layer CalcDT reads (6 planes instead of 12 for 4 cells across
// k), and the faces that no sweep fills are carried over here, from the old state. Bound by the metrics and fluxes it
// reads for the field, and on a small problem by its place in the step's chain of launches. The sweeps and the full
// update against this, steps and their output together: 32x32x4 (10 steps) 668 -> 636 us, 128x128x4 (20) 3283 -> 3184,
// 256x256x1 (20) 5298 -> 4942, 96x83x70 with FP32 fluxes (10) 4202 -> 4141. Joining the update's E2Flux and bFlux2Fld as
// well was slower (256^3: 79 us a step) and is not done.
struct PerMap {   // one axis: elements s..e of an extent n wrap; flat: 2.5D, where every layer takes the active one
    int s, e, n, nG, flat;
    __device__ __forceinline__ int wrap(int m) const { return n >= nG ? m : m % n; }   // m < nG: seldom a division
    __device__ __forceinline__ int src(int x, bool normal) const {   // normal: faces across this axis
        if (x < s) return flat ? s : e - wrap(s - x - 1);
        if (flat) return x <= s + nG ? s : x;
        const int up = normal ? 1 : 0, m = x - up - e;   // the m-th layer above
        return m >= 1 && m <= nG ? s + up + wrap(m - 1) : x;
    }
};
// what lies outside the active cells, one element more along each axis for the faces (2.5D: everything), i fastest;
// 32-bit indices (the host checks)
struct PerBox { int n[3], a0[3], na[3]; unsigned total; };
__device__ __forceinline__ void per_ijk(const PerBox& b, unsigned t, int& i, int& j, int& k) {
    const unsigned ni = b.n[0], sK = ni * b.n[1], nK = sK * (b.n[2] - b.na[2]);
    if (t < nK) {
        k = t / sK; t -= k * sK;
        if (k >= b.a0[2]) k += b.na[2];
        j = t / ni; i = t - j * ni;
        return;
    }
    t -= nK;
    const unsigned sJ = ni * b.na[2], nJ = sJ * (b.n[1] - b.na[1]);
    if (t < nJ) {
        j = t / sJ; t -= j * sJ;
        if (j >= b.a0[1]) j += b.na[1];
        k = t / ni; i = t - k * ni;
        k += b.a0[2];
        return;
    }
    t -= nJ;
    const unsigned gi = ni - b.na[0], q = t / gi;
    i = t - q * gi;
    if (i >= b.a0[0]) i += b.na[0];
    k = q / b.na[1]; j = q - k * b.na[1];
    k += b.a0[2]; j += b.a0[1];
}
__global__ void k_bc_periodic(const __grid_constant__ Lay L, const __grid_constant__ GridP g, const __grid_constant__ StateP old,
                              const __grid_constant__ StateP s,
                              const __grid_constant__ PerBox box, const __grid_constant__ PerMap mi,
                              const __grid_constant__ PerMap mj, const __grid_constant__ PerMap mk) {
    const unsigned t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= box.total) return;
    int i, j, k;
    per_ijk(box, t, i, j, k);
    // the D face's source and value; a face in the last layer across another axis belongs to no cell and carries over
    auto face = [&](int d, int ii, int jj, int kk, long long& q, bool& last) {
        const int si = mi.src(ii, d == 0), sj = mj.src(jj, d == 1), sk = mk.src(kk, d == 2);
        last = si == L.Ni || sj == L.Nj || sk == L.Nk;
        q = L.at(si, sj, sk);
        return last ? old.mf[d][q] : s.mf[d][q];
    };
    const long long c = L.at(i, j, k);
    const bool cell = i < L.Ni && j < L.Nj && k < L.Nk;
    bool put[3];
    double gas[5], lo[3], hi[3], B[3];
    const long long cs = L.at(mi.src(i, false), mj.src(j, false), mk.src(k, false));
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        long long q;
        bool last;
        lo[d] = face(d, i, j, k, q, last);
        put[d] = last || q != c;
    }
    if (cell) {
#pragma unroll
        for (int v = 0; v < 5; ++v) gas[v] = s.gas[v][cs];
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            long long q;
            bool last;
            hi[d] = face(d, i + (d == 0), j + (d == 1), k + (d == 2), q, last);
        }
        cellBxyz(L, g, lo, hi, c, B);
    }
#pragma unroll
    for (int d = 0; d < 3; ++d) if (put[d]) s.mf[d][c] = lo[d];
    if (!cell) return;
    if (cs != c) {
#pragma unroll
        for (int v = 0; v < 5; ++v) s.gas[v][c] = gas[v];
    }
#pragma unroll
    for (int x = 0; x < 3; ++x) s.b[x][c] = B[x];
}

// DivB (gridutils.F90:717-770) partial sums, one per block, reduced in a fixed order afterwards
__global__ void k_divb_partial(Lay L, GridP g, int bg, StateP s, double* partial) {
    Reg r = {L.is(), L.Nip, L.js(), L.Njp, L.ks(), L.Nkp};
    int i, j, k;
    double v = 0.0;
    if (reg_ijk(r, blockIdx.x * (long long)blockDim.x + threadIdx.x, i, j, k)) {
        long long c = L.at(i, j, k);
        double dFi = s.mf[0][c] - s.mf[0][c + 1];
        double dFj = s.mf[1][c] - s.mf[1][c + L.P];
        double dFk = s.mf[2][c] - s.mf[2][c + (long long)L.P * L.Q];
        double dFi0 = 0.0, dFj0 = 0.0, dFk0 = 0.0;
        if (bg) {   // total divergence includes the background flux (gridutils.F90:754-758)
            dFi0 = g.bFlux0[0][c] - g.bFlux0[0][c + 1];
            dFj0 = g.bFlux0[1][c] - g.bFlux0[1][c + L.P];
            dFk0 = g.bFlux0[2][c] - g.bFlux0[2][c + (long long)L.P * L.Q];
        }
        v = fabs(dFi + dFj + dFk + dFi0 + dFj0 + dFk0);
    }
    for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
    __shared__ double ws[32];
    int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (lane == 0) ws[w] = v;
    __syncthreads();
    if (w == 0) {
        int nw = blockDim.x >> 5;
        v = lane < nw ? ws[lane] : 0.0;
        for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
        if (lane == 0) partial[blockIdx.x] = v;
    }
}
__global__ void k_sum_partials(const double* partial, int n, double* out) {
    __shared__ double ws[32];
    double v = 0.0;
    for (int b = threadIdx.x; b < n; b += blockDim.x) v += partial[b];
    for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
    int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (lane == 0) ws[w] = v;
    __syncthreads();
    if (w == 0) {
        int nw = blockDim.x >> 5;
        v = lane < nw ? ws[lane] : 0.0;
        for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
        if (lane == 0) *out = v;
    }
}

// ================================================================================ host side
GridP Handle::gridP() const {
    GridP g;
    g.volume = volume;
    for (int x = 0; x < 3; ++x) g.xyzcc[x] = xyzcc[x];
    for (int d = 0; d < 3; ++d) for (int x = 0; x < 3; ++x) g.xfc[d][x] = xfc[d][x];
    g.dl = dl;
    for (int d = 0; d < 3; ++d) {
        g.face[d] = face[d]; g.edge[d] = edge[d];
        for (int q = 0; q < 9; ++q) { g.Tf[d][q] = Tf[d][q]; g.Te[d][q] = Te[d][q]; }
        for (int q = 0; q < 4; ++q) g.Teb[d][q] = Teb[d][q];
        for (int x = 0; x < 3; ++x) g.fcB0[d][x] = fcB0[d][x];
        for (int q = 0; q < 2; ++q) g.edgB0[d][q] = edgB0[d][q];
        g.B0[d] = B0[d]; g.bFlux0[d] = bFlux0[d]; g.dpB0[d] = dpB0[d];
    }
    return g;
}

static const int TPB = 128;

void mark_b_given(Handle& h, cudaStream_t st) {
    k_b_given<<<1, 1, 0, st>>>(h.dScal, B_GIVEN_STEPS);
    h.launches++;
}
void launch_b_check(Handle& h, bool n, bool o, cudaStream_t st) {
    k_b_given<<<1, 1, 0, st>>>(h.dScal, 0);
    h.launches++;
    if (!h.p.doMHD || !(n || o)) return;   // no fluxes to follow; nothing to look at
    const unsigned ny = h.L.Nk < 64 ? h.L.Nk : 64, nx = std::min(nblk((long long)h.L.Ni * h.L.Nj, TPB), 37u);   // 16 per SM
    k_b_check<<<dim3(nx, ny), TPB, 0, st>>>(h.L, h.p, h.gridP(), h.S[h.cur], h.S[h.cur ^ 1], n, o, h.dScal);
    h.launches++;
}

void launch_min_length(Handle& h, cudaStream_t st) {
    k_min_length<<<nblk(h.L.E, 256), 256, 0, st>>>(h.L.E, h.di, h.dj, h.dk, h.dl);
    h.launches++;
}

void half_planes(Handle& h, cudaStream_t st) {
    if (!h.halfDerived) return;
    h.halfDerived = false;
    if (!h.p.doBoris) {
        PrimP Wh;
        for (int v = 0; v < 5; ++v) Wh.w[v] = h.Wh[v];
        k_half_con<<<grid_plane(Reg{0, h.L.Ni, 0, h.L.Nj, 0, h.L.Nk}, TPB), TPB, 0, st>>>(h.L, h.p, Wh, h.H);
        h.launches++;
    }
    if (h.p.doMHD) {
        k_half_flux<<<nblk(h.L.E, 256), 256, 0, st>>>(h.L.E, h.gridP(), Vec3P{{h.hbA[0], h.hbA[1], h.hbA[2]}},
                                                      Vec3P{{h.H.mf[0], h.H.mf[1], h.H.mf[2]}});
        h.launches++;
    }
}

void launch_bflux2fld(Handle& h, const StateP& s, cudaStream_t st) {
    const Reg r = {0, h.L.Ni, 0, h.L.Nj, 0, h.L.Nk};
    k_bflux2fld<<<grid_plane(r, TPB), TPB, 0, st>>>(h.L, h.gridP(), s, r);
    h.launches++;
    if (h.p.doRing) launch_ring_bfix(h, s, st);   // gridutils.F90:298-300
}

void launch_bcs(Handle& h, const StateP& s, cudaStream_t st, bool withB) {
    const Lay& L = h.L;
    const int serialJ = (h.p.bc[2] == BC_LFMPOLE || h.p.bc[3] == BC_LFMPOLE) && L.Njp < L.nG;
    k_bc_i<<<dim3(nblk((long long)L.nG * (L.Nj + 1) * (L.Nk + 1), TPB), 2), TPB, 0, st>>>(L, h.p, h.gridP(), s, withB);
    if (h.p.bc[0] == BC_ION || h.p.bc[1] == BC_WIND) launch_msph_bcs(h, s, st, withB);   // IonInner, WindBC
    k_bc_j<<<dim3(nblk((long long)(L.Ni + 1) * (L.Nk + 1), TPB), serialJ ? 1 : 2 * L.nG), TPB, 0, st>>>(L, h.p, s, withB, serialJ);
    k_bc_k<<<dim3(nblk((long long)(L.Ni + 1) * (L.Nj + 1), TPB), 2 * L.nG), TPB, 0, st>>>(L, h.p, s, withB);
    h.launches += 3;
}

static PerBox per_box(const Handle& h) {
    const Lay& L = h.L;
    PerBox b = {{L.Ni + 1, L.Nj + 1, L.Nk + 1}, {L.is(), L.js(), L.ks()}, {L.Nip, L.Njp, h.p.do25D ? 0 : L.Nkp}, 0u};
    const long long n = (long long)b.n[0] * b.n[1] * b.n[2] - (long long)b.na[0] * b.na[1] * b.na[2];
    b.total = n < (1ll << 31) ? (unsigned)n : 0u;
    return b;
}
// the sides and the sizes that k_bc_periodic takes
static bool bc_in_one(const Handle& h) {
    for (int q = 0; q < 6; ++q) if (h.p.bc[q] != BC_PERIODIC) return false;
    return !h.p.doRing && !h.p.msph.on && !(h.p.do25D && h.L.Nkp > 1) && per_box(h).total > 0u;
}
static void launch_bc_periodic(Handle& h, const StateP& n, const StateP& s, cudaStream_t st) {
    const Lay& L = h.L;
    const PerBox b = per_box(h);
    const PerMap mi = {L.is(), L.ie(), L.Nip, L.nG, 0}, mj = {L.js(), L.je(), L.Njp, L.nG, 0},
                 mk = {L.ks(), L.ke(), L.Nkp, L.nG, h.p.do25D};
    k_bc_periodic<<<nblk(b.total, TPB), TPB, 0, st>>>(L, h.gridP(), n, s, b, mi, mj, mk);
    h.launches++;
}

// CalcDT's own finalization saves a launch; the many blocks of a large grid pay more for counting one another. The
// phase in us, in one launch and in two: 128x128x4 13.2 / 15.3, 64^3 (1,188 blocks) 15.2 / 17.4, 96^3 (3,724) 30.2 / 29.7,
// 128^3 51.3 / 50.2, 160^3 86.5 / 82.6, 256^3 314 / 296.
static bool dt_in_one(const Handle& h) {
    const dim3 g = grid_plane(reg_dt(h.L, h.p), 256);
    return g.x * g.y <= 2048u;
}
static void launch_calcdt_mode(Handle& h, const StateP& s, int finalize, cudaStream_t st) {
    const Lay& L = h.L;
    const bool one = dt_in_one(h);
    k_calcdt<<<grid_plane(reg_dt(L, h.p), 256), 256, 0, st>>>(L, h.p, h.gridP(), s, h.dScal, one ? finalize : -1);
    h.launches++;
    if (finalize >= 0 && !one) launch_dt_finalize(h, finalize, st);
}
void launch_calcdt_partial(Handle& h, const StateP& s, cudaStream_t st) { launch_calcdt_mode(h, s, -1, st); }

void launch_dt_finalize(Handle& h, int mode, cudaStream_t st) {
    k_dt_finalize<<<1, 1, 0, st>>>(h.p, h.dScal, mode);
    h.launches++;
}

void launch_calcdt(Handle& h, const StateP& s, int mode, cudaStream_t st) {
    launch_calcdt_mode(h, s, mode, st);
}

__global__ void k_to_f32(const double* src, float* dst, long long n) {
    long long l = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (l < n) dst[l] = float(src[l]);
}

__global__ void k_ratio_f32(const double* num, const double* den, float* dst, long long n) {
    long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (t < n) { double d = den[t]; dst[t] = d != 0.0 ? float(num[t] / d) : 0.0f; }
}

// float copies of the background planes (fcB0, bFlux0/face, edgB0)
void refresh_f32_background(Handle& h) {
    if (!h.f32pool || !h.p.doBackground) return;
    const long long E = h.L.E;
    F32Planes& f = h.f32;
    for (int d = 0; d < 3; ++d) {
        for (int x = 0; x < 3; ++x) { k_to_f32<<<nblk(E, 256), 256, 0, h.stream>>>(h.fcB0[d][x], f.fcB0[d][x], E); }
        for (int c = 0; c < 2; ++c) { k_to_f32<<<nblk(E, 256), 256, 0, h.stream>>>(h.edgB0[d][c], f.edgB0[d][c], E); }
        k_ratio_f32<<<nblk(E, 256), 256, 0, h.stream>>>(h.bFlux0[d], h.face[d], f.b0n[d], E);
        h.launches += 6;
    }
}

int ensure_f32(Handle& h) {
    if (h.f32pool) return 0;
    const long long E = h.L.E;
    const int nplanes = 28 + 24 + 64 + 6 + (h.p.doBackground ? 18 : 0);   // 6: the I and J edges' face velocities
    if (cudaMalloc(&h.f32pool, sizeof(float) * E * nplanes) != cudaSuccess) return 3;
    cudaMemsetAsync(h.f32pool, 0, sizeof(float) * E * nplanes, h.stream);
    float* q = h.f32pool;
    auto take = [&]() { float* r = q; q += E; return r; };
    F32Planes& f = h.f32;
    for (int v = 0; v < 5; ++v) f.Wh[v] = take();
    for (int v = 0; v < 5; ++v) f.Wn[v] = take();
    for (int x = 0; x < 3; ++x) f.hb[x] = take();
    for (int x = 0; x < 3; ++x) f.nb[x] = take();
    for (int x = 0; x < 3; ++x) f.hbA[x] = take();
    for (int x = 0; x < 3; ++x) f.nbA[x] = take();
    for (int x = 0; x < 3; ++x) f.Vf[x] = take();
    for (int e = 0; e < 2; ++e) for (int x = 0; x < 3; ++x) f.VfE[e][x] = take();
    for (int x = 0; x < 3; ++x) f.VdV[x] = take();
    for (int d = 0; d < 3; ++d) {
        for (int v = 0; v < 5; ++v) f.gflx[d][v] = take();
        for (int x = 0; x < 3; ++x) f.mflx[d][x] = take();
    }
    f.volume = take();
    for (int d = 0; d < 3; ++d) f.face[d] = take();
    for (int d = 0; d < 3; ++d) f.edge[d] = take();
    for (int d = 0; d < 3; ++d) for (int c = 0; c < 9; ++c) f.Tf[d][c] = take();
    for (int d = 0; d < 3; ++d) for (int c = 0; c < 6; ++c) f.Te[d][c] = take();
    for (int d = 0; d < 3; ++d) for (int c = 0; c < 4; ++c) f.Teb[d][c] = take();
    if (h.p.doBackground) {
        for (int d = 0; d < 3; ++d) {
            for (int x = 0; x < 3; ++x) f.fcB0[d][x] = take();
            for (int c = 0; c < 2; ++c) f.edgB0[d][c] = take();
            f.b0n[d] = take();
        }
    }
    auto cv = [&](const double* s_, float* d_) { k_to_f32<<<nblk(E, 256), 256, 0, h.stream>>>(s_, d_, E); h.launches++; };
    cv(h.volume, f.volume);
    for (int d = 0; d < 3; ++d) {
        cv(h.face[d], f.face[d]);
        cv(h.edge[d], f.edge[d]);
        for (int c = 0; c < 9; ++c) cv(h.Tf[d][c], f.Tf[d][c]);
        for (int c = 0; c < 6; ++c) cv(h.Te[d][3 + c], f.Te[d][c]);
        for (int c = 0; c < 4; ++c) cv(h.Teb[d][c], f.Teb[d][c]);
    }
    refresh_f32_background(h);
    return cudaGetLastError() == cudaSuccess ? 0 : 3;
}

int kernels_per_step(const Handle& h, bool split) {
    int n = 1;                          // predict cells
    if (h.p.doMHD) n += 1 + 1 + 3;      // predict faces, Mom2Face (all directions), 3 edge kernels
    n += (h.p.do25D ? 2 : 3) + ((h.fuseUpdate && !h.closure) ? 0 : 1);   // fluxes + flux2deltas
    n += 1 + 1 + 1;                     // e2flux/copy, bflux2fld, update gas
    n += (!split && dt_in_one(h) ? 1 : 2) + (!split && bc_in_one(h) ? 1 : 3 + 1);   // calcdt (+ finalize), 3 BC kernels, final bflux2fld
    n += ring_kernels_per_step(h);
    n += msph_kernels_per_step(h);
    if (h.closure) n += closure_kernels_per_step(h) + 1;   // + the conditional Flux2Deltas
    return n;
}

// NVTX ranges named after the reference's timers of the step (mhdgroup.F90:30-70, stress.F90:78-150,
// gamapp.F90:76-99): a profiler attached to an eager (non-graph) step sees its kernels under the same
// names as the reference's printClocks tree (Advance > Gamera > Predictor, E-Field, Fluxes, ...).
static const char* const kPhaseRange[NPHASE] = {"Predictor", "E-Field", "Fluxes", "Flux2Deltas", "Update", "DT",
                                                "BCs"};   // BCs is pushed by step_enqueue_bcs

// Largest problem whose kernels run beside one another. us per step with and without it, double precision / FP32 fluxes:
//   4 to 25 k cells     32x32x4 37 / 62, 64x64x1 43 / 60, 24^3 45 / 65, 41 / 54, 32x28x28 56 / 75, 44 / 57
//   33 to 51 k          32^3 72 / 88, 47 / 62, 128x64x4 82 / 89, 57 / 66, 40x40x32 99 / 107, 67 / 72
//   64 to 77 k          40^3 129 / 121, 80 / 84 (zero-gradient sides 138 / 125, 89 / 91), 128x128x4 138 / 135,
//                       96x96x8 122 / 127, 93 / 90, 48x40x40 133 / 127, 86 / 88, magnetosphere 48x42x32 226 / 228, 189 / 186
//   131 k               128x128x8 193 / 183, magnetosphere 48x42x64 315 / 322, 250 / 241
//   2.5D                256x256x1 184 / 189, 146 / 150, 312x312x1 248 / 255, 196 / 199, 512x512x1 607 / 599
//   with a closure      40^3 230 / 228, 182 / 199, 48^3 293 / 287, 243 / 250
// The graphs of a step with branches take 0.6 ms longer to set up.
static long long branch_cells(const Handle& h) { return h.p.do25D || h.closure ? 100000 : 60000; }

int step_enqueue(Handle& h, int cur, cudaEvent_t* ev, bool split, int part) {
    cudaStream_t st = h.stream;
    h.enqPrec = h.prec;
    int openRange = -1;
    auto mark = [&](int ph) {
        if (ev) cudaEventRecord(ev[ph], st);
        if (openRange >= 0) nvtxRangePop();
        openRange = ph < NPHASE ? ph : -1;
        if (openRange >= 0) nvtxRangePushA(kPhaseRange[ph]);
    };
    struct Outer {   // "Advance" around the whole enqueue, closing any open phase range on return
        int& open;
        explicit Outer(int& o) : open(o) { nvtxRangePushA("Advance"); }
        ~Outer() { if (open >= 0) nvtxRangePop(); nvtxRangePop(); }
    } outer(openRange);
    const Lay& L = h.L;
    const Par& p = h.p;
    GridP g = h.gridP();
    StateP nS = h.S[cur], oS = h.S[cur ^ 1];
    // The fluxes and the E field, and the two predictors, run beside one another where they are far from filling the GPU:
    // a step is a chain of dependent launches, and a small problem's step costs the length of that chain. Not in larger
    // problems, which gain nothing and pay for the joins (branch_cells), and not where other problems' steps run beside
    // this one (a 24-member ensemble's 20 steps 2.23 -> 2.31 ms with branches).
    Branches br(st, ev == nullptr && h.alone && (long long)L.Nip * L.Njp * L.Nkp <= branch_cells(h));
    const float* corr = nullptr;
    // what the update writes: everything, or, where k_bc_periodic writes all that lies further out, the active cells and
    // the layer around them that CalcDT reads
    const bool one = !split && bc_in_one(h);
    const Reg cells = one ? Reg{L.is() - 1, L.Nip + 2, L.js() - 1, L.Njp + 2, L.ks() - 1, L.Nkp + 2}
                          : Reg{0, L.Ni, 0, L.Nj, 0, L.Nk};
    const Reg faces = {cells.i0, cells.ni + 1, cells.j0, cells.nj + 1, cells.k0, cells.nk + 1};
    const Reg act = {L.is(), L.Nip, L.js(), L.Njp, L.ks(), L.Nkp};
    if (part != STEP_POST) {
    mark(PH_PREDICT);
    // learned closure: face corrections from the net on State n, needed by Flux2Deltas, whose phase they are timed with
    if (h.closure && part == STEP_ALL && !ev) {
        br.go(SIDE_NET);
        if (int rc = closure_enqueue_corr(h, nS, st, &corr)) return rc;
        br.back();
    }
    if (p.doMHD) {
        Vec3P mf = {{nS.mf[0], nS.mf[1], nS.mf[2]}}, omf = {{oS.mf[0], oS.mf[1], oS.mf[2]}},
              hmf = {{h.H.mf[0], h.H.mf[1], h.H.mf[2]}}, hbA = {{h.hbA[0], h.hbA[1], h.hbA[2]}},
              nbA = {{h.nbA[0], h.nbA[1], h.nbA[2]}};
        F32FaceOut fo{};
        if (h.prec == PREC_FP32FLUX)
            for (int x = 0; x < 3; ++x) { fo.hbA[x] = h.f32.hbA[x]; fo.nbA[x] = h.f32.nbA[x]; }
        br.go(SIDE_FLUX);
        k_predict_faces<<<nblk(L.E / 2, 256), 256, 0, st>>>(L.E, p, g, mf, omf, hmf, hbA, nbA, fo, h.dScal);
        br.back();
        h.launches++;
    }
    PrimP Wh, Wn;
    for (int v = 0; v < 5; ++v) { Wh.w[v] = h.Wh[v]; Wn.w[v] = h.Wn[v]; }
    F32CellOut fc{};
    if (h.prec == PREC_FP32FLUX) {
        for (int v = 0; v < 5; ++v) { fc.Wh[v] = h.f32.Wh[v]; fc.Wn[v] = h.f32.Wn[v]; }
        for (int x = 0; x < 3; ++x) { fc.hb[x] = h.f32.hb[x]; fc.nb[x] = h.f32.nb[x]; fc.VdV[x] = h.f32.VdV[x]; }
    }
    k_predict_cells<<<grid_plane(Reg{0, L.Ni, 0, L.Nj, 0, L.Nk}, TPB), TPB, 0, st>>>(L, p, g, nS, oS, h.H, Wh, Wn, fc, h.dScal);
    h.launches += 1;
    if (p.doRing) launch_ring_bfix(h, h.H, st, h.prec == PREC_FP32FLUX);   // bFlux2Fld's ring fix
    if (p.predFixLFM) launch_predfix_lfm(h, h.H, st, h.prec == PREC_FP32FLUX);   // HackPredictor
    if (p.doMHD) br.join(SIDE_FLUX);
    mark(PH_EFIELD);
    // the flux kernels beside the E field's (after it where everything is on one stream)
    if (br.on && part == STEP_ALL) enqueue_fluxes(h, nS, br);
    if (p.doMHD) {
        enqueue_efield(h, nS, br);
        if (p.msph.on) launch_msph_efix(h, nS, st);   // HackE (mhdgroup.F90:40-44)
    }
    if (br.on && part == STEP_ALL)
        for (int d = 0; d < (p.do25D ? 2 : 3); ++d) br.join(SIDE_FLUX + d);
    }
    if (part == STEP_PRE) return (int)cudaGetLastError();
    if (part == STEP_ALL && !br.on) {
        mark(PH_FLUXES);
        enqueue_fluxes(h, nS, br);
    }
    if (p.doRing) launch_ring_flux(h, st);   // stress.F90:134-139
    if (p.msph.on) launch_ion_flux(h, st);    // HackFlux (stress.F90:141-143)
    mark(PH_DELTAS);
    PrimP dGH;
    for (int v = 0; v < 5; ++v) dGH.w[v] = h.dGasH[v];
    Vec3P dGM = {{h.dGasM[0], h.dGasM[1], h.dGasM[2]}};
    FluxOut<float> F32[3];
    FluxP F64[3];
    for (int d = 0; d < 3; ++d) {
        for (int v = 0; v < 5; ++v) { F32[d].g[v] = h.f32.gflx[d][v]; F64[d].g[v] = h.gflx[d][v]; }
        for (int x = 0; x < 3; ++x) { F32[d].m[x] = h.f32.mflx[d][x]; F64[d].m[x] = h.mflx[d][x]; }
    }
    // without a closure the update computes the deltas itself (no dGasH/dGasM round trip through HBM)
    const bool fuse = h.fuseUpdate && !h.closure;
    // learned closure: a corrected update that fails positivity falls back to the plain fluxes (the second, conditional
    // Flux2Deltas). With the ensembles' tile queue, and timed by phases, the net runs here.
    if (corr) br.join(SIDE_NET);
    else if (h.closure)
        if (int rc = closure_enqueue_corr(h, nS, st, &corr)) return rc;
    for (int pass = 0; pass < (fuse ? 0 : (corr ? 2 : 1)); ++pass) {
        const float* cq = pass == 0 ? corr : nullptr;
        const Scal* cond = pass == 0 ? nullptr : h.dScal;
        if (h.prec == PREC_FP32FLUX)
            k_flux2deltas<float><<<grid_plane(act, TPB), TPB, 0, st>>>(L, p, g, F32[0], F32[1], F32[2], dGH, dGM, cq, cond);
        else
            k_flux2deltas<double><<<grid_plane(act, TPB), TPB, 0, st>>>(L, p, g, F64[0], F64[1], F64[2], dGH, dGM, cq, cond);
        if (pass == 0 && corr) closure_enqueue_check(h, nS, st);
        if (pass == 1) h.launches++;
    }
    mark(PH_UPDATE);
    // applyUpdate into the oState buffer (which becomes State n+1); only the Boris update needs the new field
    Vec3P E = {{h.E[0], h.E[1], h.E[2]}};
    const bool apart = !p.doBoris;
    auto update = [&](cudaStream_t us) {
        const dim3 gc = grid_plane(cells, TPB);
        if (h.prec == PREC_FP32FLUX) {
            if (fuse) k_update_gas<float, true><<<gc, TPB, 0, us>>>(L, p, g, nS, oS, dGH, dGM, F32[0], F32[1], F32[2], cells, h.dScal);
            else k_update_gas<float, false><<<gc, TPB, 0, us>>>(L, p, g, nS, oS, dGH, dGM, F32[0], F32[1], F32[2], cells, h.dScal);
        } else {
            if (fuse) k_update_gas<double, true><<<gc, TPB, 0, us>>>(L, p, g, nS, oS, dGH, dGM, F64[0], F64[1], F64[2], cells, h.dScal);
            else k_update_gas<double, false><<<gc, TPB, 0, us>>>(L, p, g, nS, oS, dGH, dGM, F64[0], F64[1], F64[2], cells, h.dScal);
        }
    };
    if (apart) {
        br.go(SIDE_FLUX);
        update(st);
        br.back();
    }
    if (p.doRing && p.doMHD) launch_pole_e(h, h.E, st);   // mhdgroup.F90:139-142
    if (h.closure && p.doMHD) closure_enqueue_emf(h, st);
    k_e2flux<<<grid_plane(faces, TPB), TPB, 0, st>>>(L, p, E, nS, oS, faces, h.dScal);
    // bFlux2Fld of the update; with ring averaging its ring fix is left to the RingAverage bFlux2Fld,
    // which recomputes every cell before anything reads a ghost B
    if (p.doMHD) k_bflux2fld<<<grid_plane(cells, TPB), TPB, 0, st>>>(L, g, oS, cells);
    else k_copy_b<<<nblk(L.E, 256), 256, 0, st>>>(L, nS, oS);
    if (!apart) update(st);
    else br.join(SIDE_FLUX);
    h.launches += 3;
    if (p.msph.on) launch_apply_grav(h, oS, nS, st);   // mhdgroup.F90:60-65 (oS holds the new state)
    if (p.doRing) launch_ring_average(h, oS, st);   // mhdgroup.F90:68-74
    if (p.msph.on) launch_msph_perstep(h, oS, st);   // HackStep (gamapp.F90:104-109)
    // CalcDT (the per-cell minimum; finalized below, or after the tiles' minimum for a tiled run)
    mark(PH_DT);
    launch_calcdt_mode(h, oS, split ? -1 : 0, st);
    if (!split) {
        if (one) {
            mark(PH_BCS);
            launch_bc_periodic(h, nS, oS, st);
        } else {
            step_enqueue_bcs(h, cur, ev, true);
            step_enqueue_ghosts(h, cur);
        }
        mark(NPHASE);
    }
    const int rc = (int)cudaGetLastError();
    return rc == 0 && br.failed ? -1 : rc;
}

// The rest of CalcDT, then EnforceBCs on the new state S[cur ^ 1]
void step_enqueue_bcs(Handle& h, int cur, cudaEvent_t* ev, bool finalized) {
    cudaStream_t st = h.stream;
    if (!finalized) launch_dt_finalize(h, 0, st);
    if (ev) cudaEventRecord(ev[PH_BCS], st);
    nvtxRangePushA("BCs");
    launch_bcs(h, h.S[cur ^ 1], st, false);   // step_enqueue_ghosts rewrites every ghost B
    nvtxRangePop();
}

// bFlux2Fld of the ghost cells of the new state S[cur ^ 1], after the BCs (and the halo fill of a tile)
void step_enqueue_ghosts(Handle& h, int cur) {
    cudaStream_t st = h.stream;
    const Lay& L = h.L;
    StateP s = h.S[cur ^ 1];
    if (h.p.do25D) launch_bflux2fld(h, s, st);   // the 2.5D K replication rewrites an active cell's upper face
    else {
        k_bflux2fld_ghost<<<nblk(ghost_cells(L), TPB), TPB, 0, st>>>(L, h.gridP(), s);
        h.launches++;
        if (h.p.doRing) launch_ring_bfix(h, s, st);
    }
}

double launch_divb(Handle& h, double* scratchDev, cudaStream_t st) {
    const Lay& L = h.L;
    long long n = (long long)L.Nip * L.Njp * L.Nkp;
    int nb = (int)nblk(n, 256);
    StateP s = h.S[h.cur];
    k_divb_partial<<<nb, 256, 0, st>>>(L, h.gridP(), h.p.doBackground, s, scratchDev);
    k_sum_partials<<<1, 1024, 0, st>>>(scratchDev, nb, scratchDev + nb);
    h.launches += 2;
    double out = 0.0;
    cudaMemcpyAsync(&out, scratchDev + nb, sizeof(double), cudaMemcpyDeviceToHost, st);
    cudaStreamSynchronize(st);
    return out;
}

}  // namespace gam
