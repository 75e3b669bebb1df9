// Per-stage kernels of the ES-DGSEM engine (sm_100a, FP64).
//
// One RK stage of the plain path is two launches:
//   face_flux  : one thread per face node gathers the two traces straight
//                from q (wall ghost on boundary faces), evaluates the ES
//                Riemann flux once and writes it to both elements' sides;
//   element    : (esdg_tma.cuh, esdg_pair.cuh or esdg_oneshot.cuh, by the
//                rule of Engine::rule_variant; esdg_rows.cuh where a caller
//                fixes its variants) flux-
//                differencing volume integral, lifting of the four face
//                fluxes, low-storage (or SSP) RK update and, on the last
//                stage, the element wave-speed maximum for the next dt.
// With artificial viscosity (BR1 gradient + viscous terms) a stage is the
// sensor pass (esdg_indicator.cuh; at the step start and before stages > 0),
// which flags the elements whose viscous terms are not exactly zero, then
// face_flux (+ gradient face flux of their faces), element (updates the
// others, writes Qt of the flagged ones and lists them), and over the list
// grad_list (lifted BR1 gradient) and viscous_list (viscous face fluxes,
// volume and lift + RK update).  A stage of a 256x256 dam break, N = 4, 1.4 %
// of the elements viscous: 121 us, against 241 with the viscous terms formed
// everywhere; with every element viscous 246 against 249.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "esdg_physics.cuh"
#include "esdg_partialdry.cuh"

namespace esdg {

enum : int { ST_OK = 0, ST_NONFINITE = 1 };

// Per-instance time-stepping state, resident in device memory so that a
// whole step runs without a host round trip (and can be graph-captured).
struct DevState {
    double t, dt, T, minEle, CFL, DFL;
    unsigned long long lam_key, visc_key;
    int steps, max_steps, done, status;
    // checkpoint pause (pause_on != 0): a step does not start once t >=
    // pause_at and at least one step ran since steps == resume_steps; the
    // host writes its outputs and resumes (the reference's plot checkpoints,
    // src/deviceclass.cpp:1143-1147, one per step)
    double pause_at;
    int pause_on, resume_steps;
};

// Element-side face fluxes (the SP buffer of the engine): for side s of
// element e, the scaled ES flux of that side's face at the side's own nodes
// j = 0..NGL-1 (the element's orientation of the side), already multiplied
// by -MasterSlave: SP[((e * 4 + s) * 3 + eq) * NGL + j].  The element then
// adds fs * Jinv, which is the reference's -ms * flux * Jinv
// (okl/DG/SurfaceKernel.okl:17-142) bit for bit (the sign flip is exact),
// and bulk-copies its tile's fluxes with the rest of the tile.
__host__ __device__ __forceinline__ long side_flux_at(int e, int side, int eq, int j, int ngl) {
    return ((long)(e * 4 + side) * 3 + eq) * ngl + j;
}

// Packed face record: x elemL, y elemR or -1, z sideL | sideR << 2 |
// sameOrient << 4, w the element-side flags the face kernel needs to write
// element-side fluxes: orientation of the left side (bit 0), its
// MasterSlave == -1 (bit 1), the same two for the right side (bits 2, 3).
__host__ __device__ __forceinline__ int face_side_flags(int orientL, int msL, int orientR, int msR) {
    return (orientL ? 1 : 0) | (msL < 0 ? 2 : 0) | (orientR ? 4 : 0) | (msR < 0 ? 8 : 0);
}

struct FaceArgs {
    int F;
    const int4* __restrict__ ftab;  // (elemL, elemR or -1, sideL | sideR<<2 | sameOrient<<4, side flags)
    const double* __restrict__ q;
    const double* __restrict__ nx;
    const double* __restrict__ ny;
    const double* __restrict__ scal;
    const double* __restrict__ bL;
    const double* __restrict__ bR;
    double* __restrict__ SP;   // element-side fluxes [K][4][3][ngl]
    double* __restrict__ SGX;  // [F][2][ngl] (AV only)
    double* __restrict__ SGY;
    const int* __restrict__ elem_inst;
    const DevState* __restrict__ st;
    PhysConst c;
    // active set (AV): gradient fluxes only where an adjacent element is
    // flagged
    const int* __restrict__ act = nullptr;
    // live extent (null: all): [0] elements, [1] faces below which every
    // live entity lies (the arena keeps it current between replays)
    const int* __restrict__ extent = nullptr;
    // Testcase 1 (conv = 1): exact outer states on boundary faces at the
    // stage time t + tfrac dt, from the nodal coordinates X, Y
    int conv = 0;
    double tfrac = 0.0;
    const double* __restrict__ X = nullptr;
    const double* __restrict__ Y = nullptr;
};

struct ElemArgs {
    int K;
    const double* __restrict__ Jinv;
    const double* __restrict__ Yxi;
    const double* __restrict__ Yeta;
    const double* __restrict__ Xxi;
    const double* __restrict__ Xeta;
    const double* __restrict__ Bx;
    const double* __restrict__ By;
    const double* __restrict__ B;
    const double* __restrict__ D;       // flux-differencing matrix [ngl][ngl]
    const double* __restrict__ Dhat;    // BR1 gradient matrix
    const double* __restrict__ Dstrong; // viscous volume matrix
    const double* __restrict__ Vinv;    // modal transform
    const double* __restrict__ SP;      // element-side face fluxes [K][4][3][ngl] (see side_flux_at)
    const double* __restrict__ SGX;     // gradient face fluxes [F][2][ngl]
    const double* __restrict__ SGY;
    const int4* __restrict__ ftab;      // faces, as in FaceArgs (viscous face flux)
    const double* __restrict__ nx;
    const double* __restrict__ ny;
    const double* __restrict__ scal;
    const int4* __restrict__ side;      // per element side: (face, masterSlave, orientation, 0)
    double* q;
    double* __restrict__ gRK;
    double* __restrict__ Qt;
    const double* __restrict__ Qtmp;
    double* __restrict__ GX;            // [K][2][ngl][ngl]
    double* __restrict__ GY;
    double* __restrict__ VP;            // [K]
    const int* __restrict__ elem_inst;
    DevState* st;
    double rkA, rkB, rkC;
    int mode;        // 0: LS-RK update, 1: SSP update, 2: write Qt only
    int lam;         // 1: element wave speed max into st[inst].lam_key after the update
    PhysConst c;
    // Active set (null: none).  Plain element kernels write Qt instead of
    // updating flagged elements and append them to alist (count in
    // *acount); k_grad_list and k_viscous_list then run over alist only.
    // clear_act: k_viscous_list takes the flags back.
    int* act = nullptr;
    int clear_act = 0;
    int* alist = nullptr;
    int* acount = nullptr;
    const int* __restrict__ extent = nullptr;  // live extent, as in FaceArgs
    // Partial-dry treatment (null: off): per-element dry flag, nodal b, and
    // the central / forward / backward difference matrices [n*n].
    const int* __restrict__ dry = nullptr;
    const double* __restrict__ Bn = nullptr;
    const double* __restrict__ Dc = nullptr;
    const double* __restrict__ Dup = nullptr;
    const double* __restrict__ Ddn = nullptr;
    // Testcase 1 (conv = 1): the manufactured source at the stage time
    // t + tfrac dt from the nodal coordinates X, Y (b: B, its derivatives:
    // Bx, By)
    int conv = 0;
    double tfrac = 0.0;
    const double* __restrict__ X = nullptr;
    const double* __restrict__ Y = nullptr;
    // Bounded waits of the bulk-copy kernels: limit in clock cycles (0: the
    // default, about 2 s) and, for a test of the timeout path, a tile whose
    // copies are never issued (tile + 1; 0: none).  Zero-initialised
    // arguments leave both off.
    long long wait_limit = 0;
    int skip_tile = 0;
};

// r += the manufactured source of node xid (Testcase 1).
__device__ __forceinline__ void add_conv_source(const ElemArgs& a, const DevState& S, long xid, double Bx, double By,
                                                double& r0, double& r1, double& r2) {
    double s0, s1, s2;
    conv_source(a.c.g, a.X[xid], a.Y[xid], S.t + a.tfrac * S.dt, Bx, By, a.B[xid], s0, s1, s2);
    r0 += s0;
    r1 += s1;
    r2 += s2;
}

__device__ __forceinline__ int inst_of(const int* elem_inst, int e) { return elem_inst ? elem_inst[e] : 0; }

// Appends the tile's flagged live elements e0 .. e0 + n - 1 to the list: one
// atomic per warp of elements (the list's order does not matter, but an
// atomic per flagged element on one counter is a serial chain where the
// whole mesh is flagged).  By one whole warp of the block.
__device__ __forceinline__ void list_tile(const ElemArgs& a, int e0, int n) {
    const int lane = threadIdx.x & 31;
    for (int b = 0; b < n; b += 32) {
        const int e = e0 + b + lane;
        const bool on = b + lane < n && e < a.K && a.act[e] != 0 && !a.st[inst_of(a.elem_inst, e)].done;
        const unsigned m = __ballot_sync(0xffffffffu, on);
        if (m == 0) continue;
        int base = 0;
        if (lane == 0) base = atomicAdd(a.acount, __popc(m));
        base = __shfl_sync(0xffffffffu, base, 0);
        if (on) a.alist[base + __popc(m & ((1u << lane) - 1u))] = e;
    }
}

// ---------------------------------------------------------------------------
// Face kernel.
// ---------------------------------------------------------------------------
// One face node (gid = face * NGL + node) of the face kernel.
template <int NGL, int NUMFLUX, bool AV, bool WAIT>
__device__ __forceinline__ void face_flux_node(const FaceArgs& a, long gid) {
    const int f = (int)(gid / NGL), i = (int)(gid % NGL);
    constexpr int N2 = NGL * NGL;
    const int4 t = a.ftab[f];
    // the face's own data does not depend on the table entry: requested
    // together with it, ahead of the instance check
    const long ex = (long)f * NGL + i;
    const double nx = a.nx[ex], ny = a.ny[ex], sc = a.scal[ex], bLx = a.bL[ex];
    const int eL = t.x, eR = t.y, sL = t.z & 3, sR = (t.z >> 2) & 3, same = (t.z >> 4) & 1;
    if (WAIT) pdl_wait();  // the table and the geometry are constant, the state is the previous kernel's
    // the instance's done flag (behind the instance table in an arena) is
    // requested together with the traces, not before them: a face of a
    // finished instance reads valid memory and stores nothing
    const DevState& S = a.st[inst_of(a.elem_inst, eL)];
    const int ir = same ? i : NGL - 1 - i;
    const double* qe = a.q + (long)eL * 3 * N2;
    const int oL = trace_offset(sL, i, NGL);
    const double hL = qe[oL], huL = qe[oL + N2], hvL = qe[oL + 2 * N2];
    double hR, huR, hvR;      // right state at master node i (flux)
    double ghR, ghuR, ghvR;   // right state at node i in the right element's order (gradient)
    const bool grad = AV && (a.act[eL] || (eR >= 0 && a.act[eR]));
    if (eR >= 0) {
        const double* qr = a.q + (long)eR * 3 * N2;
        const int o = trace_offset(sR, ir, NGL);
        hR = qr[o]; huR = qr[o + N2]; hvR = qr[o + 2 * N2];
        if (grad) {
            const int o2 = trace_offset(sR, i, NGL);
            ghR = qr[o2]; ghuR = qr[o2 + N2]; ghvR = qr[o2 + 2 * N2];
        }
    } else {
        // The reference stores the ghost of every face node in order and reads
        // it back at node ir (okl/GatherEdgeData/SolidWalls.okl:150-173).
        const long exr = (long)f * NGL + ir;
        const int o = trace_offset(sL, ir, NGL);
        if (a.conv) {  // okl/GatherEdgeData/Dirichlet_ConvTest.okl:112-119, read back the same way
            const long xo = (long)eL * N2 + o;
            conv_exact(a.X[xo], a.Y[xo], S.t + a.tfrac * S.dt, a.bL[exr], hR, huR, hvR);
        } else {
            wall_ghost(a.nx[exr], a.ny[exr], qe[o], qe[o + N2], qe[o + 2 * N2], hR, huR, hvR);
        }
        if (grad) { ghR = hL; ghuR = huL; ghvR = hvL; }
    }
    const double bRx = a.bR[(long)f * NGL + ir];
    if (S.done) return;
    double N0, N1, N2f;
    es_flux<NUMFLUX>(a.c, nx, ny, hL, huL, hvL, hR, huR, hvR, bLx, bRx, N0, N1, N2f);
    const double s = sc;
    const double v0 = s * a.c.geomFace * N0, v1 = s * a.c.geomFace * N1, v2 = s * a.c.geomFace * N2f;
    // both sides' copies, each in its element's node order and signed by
    // -MasterSlave (side_flux_at)
    const int w = t.w;
    const int jL = (w & 1) ? i : NGL - 1 - i;
    double* pl = a.SP + side_flux_at(eL, sL, 0, jL, NGL);
    const bool nL = (w & 2) != 0;
    pl[0] = nL ? v0 : -v0; pl[NGL] = nL ? v1 : -v1; pl[2 * NGL] = nL ? v2 : -v2;
    if (eR >= 0) {
        const int jR = (w & 4) ? i : NGL - 1 - i;
        double* pr = a.SP + side_flux_at(eR, sR, 0, jR, NGL);
        const bool nR = (w & 8) != 0;
        pr[0] = nR ? v0 : -v0; pr[NGL] = nR ? v1 : -v1; pr[2 * NGL] = nR ? v2 : -v2;
    }
    if (grad) {
        // okl/BR1_Gradient/calcNumFluxesGradient.okl:16-135 (the right trace
        // is taken in the right element's own order, as there).
        const double tol = a.c.PosPresTOL;
        const double iL = (hL > tol) ? 1.0 / hL : 0.0;
        const double iR = (ghR > tol) ? 1.0 / ghR : 0.0;
        const double uL = huL * iL, uR = ghuR * iR, vL = hvL * iL, vR = ghvR * iR;
        double* gx = a.SGX + (long)f * 2 * NGL + i;
        double* gy = a.SGY + (long)f * 2 * NGL + i;
        gx[0] = nx * s * a.c.geomFace * 0.5 * (uL + uR);
        gx[NGL] = nx * s * a.c.geomFace * 0.5 * (vL + vR);
        gy[0] = ny * s * a.c.geomFace * 0.5 * (uL + uR);
        gy[NGL] = ny * s * a.c.geomFace * 0.5 * (vL + vR);
    }
}

// STRIDE = false: one thread per face node (a single mesh's one-shot
// grid).  STRIDE = true: a resident grid strides over the face nodes below
// the live extent (an arena, whose face capacity can be far above its live
// faces); a separate instantiation, since the loop costs registers.
template <int NGL, int NUMFLUX, bool AV, bool STRIDE = false>
__global__ void __launch_bounds__(256, STRIDE ? 4 : 1) k_face_flux(FaceArgs a) {
    pdl_release();
    long gid = (long)blockIdx.x * blockDim.x + threadIdx.x;
    const long all = (long)a.F * NGL;
    if (!STRIDE) {
        // Descending face order.  Face ids follow the element order (a face
        // is numbered by the first element that has it) and the element
        // kernels walk their tiles upwards, so the first faces taken here
        // read the traces the element kernel wrote last, and the fluxes
        // written last are those of the first tiles the next element kernel
        // reads: both still in L2.
        const long n = a.extent ? min(all, (long)a.extent[1] * NGL) : all;
        if (gid >= n) return;
        face_flux_node<NGL, NUMFLUX, AV, true>(a, n - 1 - gid);
    } else {
        const long n = a.extent ? min(all, (long)a.extent[1] * NGL) : all;
        pdl_wait();
        for (; gid < n; gid += (long)gridDim.x * blockDim.x) face_flux_node<NGL, NUMFLUX, AV, false>(a, gid);
    }
}

// ---------------------------------------------------------------------------
// Element kernels.
// ---------------------------------------------------------------------------
template <int NGL>
struct ElemShape {
    static constexpr int N2 = NGL * NGL;
    static constexpr int NE = (256 / N2) > 0 ? (256 / N2) : 1;  // elements per block
    static constexpr int THREADS = NE * N2;
};

// Wave-speed maximum folded into the owning instance's key
// (okl/DG/FindLambdaMax.okl:17-100 per node; a max, so the reduction order
// does not matter).  Warp-level and barrier-free: a shuffle reduction and
// one atomic per warp when all its lanes belong to one instance (always for
// a single mesh), one atomic per lane otherwise.  Must be called by every
// thread of the block (THREADS threads, the last warp possibly partial).
template <int THREADS>
__device__ __forceinline__ void warp_lambda(double lam, bool valid, int ins, DevState* st) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nl = (warp == (THREADS - 1) / 32 && (THREADS % 32) != 0) ? (THREADS % 32) : 32;
    const unsigned mask = (nl == 32) ? 0xffffffffu : ((1u << nl) - 1u);
    const int my = valid ? ins : -1;
    const int top = __reduce_max_sync(mask, my);
    if (top < 0) return;  // no valid lane in this warp
    const int low = -__reduce_max_sync(mask, valid ? -ins : -0x7fffffff);
    if (low == top) {
        double v = valid ? lam : 0.0;
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
            const double o = __shfl_down_sync(mask, v, off);
            if (lane + off < nl) v = (isnan(o) || o > v) ? o : v;
        }
        if (lane == 0) atomicMax(&st[top].lam_key, dbl_key(v));
    } else if (valid) {
        atomicMax(&st[ins].lam_key, dbl_key(lam));
    }
}

__device__ __forceinline__ double node_lambda(const PhysConst& c, double h, double hu, double hv) {
    const double inv = (h > c.PosPresTOL) ? 1.0 / h : 0.0;
    const double cc = sqrt(c.g * h);
    return cc + fmax(fabs(hu * inv), fabs(hv * inv));
}

// Tail of the modal energy sensor (okl/ShockCapturing/ShockCapturing.okl:131-227):
// energy ratios of the highest modes from the modal coefficients w
// [mode_xi][mode_eta], log10, and the sine ramp between sigma_min and
// sigma_max.  Sums in the reference's order.
template <int NGL, int S = NGL>
__device__ double sensor_tail(const PhysConst& c, const double* w) {  // w[i * S + j]
    constexpr int N = NGL - 1;
    double z1 = 0, n1 = 0, z2 = 0, n2s = 0;
    for (int i = 0; i < N; ++i) z1 += w[i * S + N] * w[i * S + N] + w[N * S + i] * w[N * S + i];
    z1 += w[N * S + N] * w[N * S + N];
    for (int i = 0; i < N - 1; ++i)
        z2 += w[i * S + N - 1] * w[i * S + N - 1] + w[(N - 1) * S + i] * w[(N - 1) * S + i];
    z2 += w[(N - 1) * S + N - 1] * w[(N - 1) * S + N - 1];
    for (int i = 0; i < NGL; ++i)
        for (int j = 0; j < NGL; ++j) n1 += w[i * S + j] * w[i * S + j];
    for (int i = 0; i < N; ++i)
        for (int j = 0; j < N; ++j) n2s += w[i * S + j] * w[i * S + j];
    const double t1 = (n1 < c.ZeroTOL) ? 0.0 : z1 / n1;
    const double t2 = (n1 < c.ZeroTOL) ? 0.0 : z2 / n2s;
    const double ratio = (t1 < t2) ? t2 : t1;
    // exact shortcut: log10 is accurate to an ulp, so below this bound the
    // reference's test sigmaMin >= log10(ratio) holds (NaN falls through)
    if (ratio < c.sensor_skip) return 0.0;
    if (ratio > c.sensor_full) return c.eps0;
    const double sig = log10(ratio);
    if (c.sigmaMin >= sig) return 0.0;
    if (c.sigmaMax >= sig) {
        const double delta = 1.0 + sin(M_PI * (sig - 0.5 * (c.sigmaMax + c.sigmaMin)) / (c.sigmaMax - c.sigmaMin));
        return c.eps0 * 0.5 * delta;
    }
    return c.eps0;
}

// Modal transform entries of the sensor: M1[i][j] = sum_l V[i][l] m[j][l]
// and w[i][j] = sum_l M1[i][l] V[j][l] (s_Q1modal[i][j] of the reference
// holds node (xi=i, eta=j)); one entry per call, so that a thread per entry
// computes exactly what the serial loops do.
template <int NGL>
__device__ __forceinline__ double sensor_m1(const double* V, const double* m, int i, int j) {
    double acc = 0.0;
    for (int l = 0; l < NGL; ++l) acc += V[i * NGL + l] * m[j * NGL + l];
    return acc;
}
template <int NGL>
__device__ __forceinline__ double sensor_w(const double* V, const double* M1, int i, int j) {
    double acc = 0.0;
    for (int l = 0; l < NGL; ++l) acc += M1[i * NGL + l] * V[j * NGL + l];
    return acc;
}

// Viscous volume term + viscous lift added to Qt, then the RK update, of the
// elements of alist[0 .. *acount), a grid-stride loop over tiles of NE list
// entries.
// okl/ViscoseParts/VolumeKernelViscose.okl:17-150, SurfaceKernelVisc.okl:17-144;
// the viscous face flux (okl/BR1_Gradient/CollectEdgeDataGradient.okl:17-194,
// okl/ViscoseParts/calcNumFluxesViscose.okl:17-107; zero on walls) is formed
// by each of the face's two elements at its own node: a dozen operations on
// four gathered values, cheaper than a kernel of its own and its flux array.
// Where neither side has viscosity it is exactly zero and the neighbour (whose
// gradient need not exist) is not read.
template <int NGL>
__global__ void __launch_bounds__(ElemShape<NGL>::THREADS) k_viscous_list(ElemArgs a) {
    constexpr int N2 = NGL * NGL, NE = ElemShape<NGL>::NE;
    __shared__ double sDs[N2];
    __shared__ double sF2[NE * N2], sF3[NE * N2], sG2[NE * N2], sG3[NE * N2];
    const int tid = threadIdx.x;
    const int el = tid / N2, nd = tid % N2;
    const int xi = nd % NGL, eta = nd / NGL;
    const int s = el * N2 + nd;
    // the node's sides (-1: none) and its place along them
    const int sn[2] = {eta == 0 ? 0 : (eta == NGL - 1 ? 2 : -1), xi == NGL - 1 ? 1 : (xi == 0 ? 3 : -1)};
    const int jn[2] = {xi, eta};
    if (tid < N2) sDs[tid] = a.Dstrong[tid];
    pdl_wait();
    const int count = *a.acount;
    for (int t = blockIdx.x; t * NE < count; t += gridDim.x) {
        if ((t + gridDim.x) * NE >= count) pdl_release();  // the CTA's last tile
        const int idx = t * NE + el;
        const bool active = idx < count;  // listed elements are live
        const int e = active ? a.alist[idx] : 0;
        const int ins = active ? inst_of(a.elem_inst, e) : 0;
        const long xid = (long)e * N2 + nd, qid = (long)e * 3 * N2 + nd, gid = (long)e * 2 * N2 + nd;
        int4 sd[2], fc[2];
        double f0[2] = {0.0, 0.0}, f1[2] = {0.0, 0.0};
        int ms[2] = {0, 0};
        if (active) {
#pragma unroll
            for (int pass = 0; pass < 2; ++pass) sd[pass] = sn[pass] >= 0 ? a.side[(long)e * 4 + sn[pass]] : int4{};
            const double eps = a.VP[e];
#pragma unroll
            for (int pass = 0; pass < 2; ++pass) fc[pass] = sn[pass] >= 0 ? a.ftab[sd[pass].x] : int4{};
            const double F2 = eps * a.GX[gid], F3 = eps * a.GX[gid + N2];
            const double G2 = eps * a.GY[gid], G3 = eps * a.GY[gid + N2];
            const double ye = a.Yeta[xid], yx = a.Yxi[xid], xe = a.Xeta[xid], xx = a.Xxi[xid];
            sF2[s] = ye * F2 - xe * G2;
            sG2[s] = -yx * F2 + xx * G2;
            sF3[s] = ye * F3 - xe * G3;
            sG3[s] = -yx * F3 + xx * G3;
            // face fluxes of the node's sides, ahead of the barrier: their
            // chain of gathers runs while the tile's other loads do
#pragma unroll
            for (int pass = 0; pass < 2; ++pass) {
                if (sd[pass].y == 0) continue;
                const int i = sd[pass].z ? jn[pass] : NGL - 1 - jn[pass];  // the face's node
                const int sL = fc[pass].z & 3, sR = (fc[pass].z >> 2) & 3, same = (fc[pass].z >> 4) & 1;
                const bool left = fc[pass].x == e && sL == sn[pass];
                const int o = left ? fc[pass].y : fc[pass].x;
                double N0 = 0.0, N1 = 0.0;
                const double vm = o >= 0 ? fmax(eps, a.VP[o]) : 0.0;
                const long ex = (long)sd[pass].x * NGL + i;
                const double sc = a.scal[ex];
                if (!(vm <= 0.0)) {
                    // traces of the face's node: the left side's i, the right side's i or its mirror
                    const int tL = trace_offset(sL, i, NGL), tR = trace_offset(sR, same ? i : NGL - 1 - i, NGL);
                    const long og = (long)o * 2 * N2 + (left ? tR : tL);
                    const long mg = (long)e * 2 * N2 + (left ? tL : tR);  // this thread's node on most meshes
                    const double nx = a.nx[ex], ny = a.ny[ex];
                    N0 = 0.5 * vm * ((nx * a.GX[mg] + ny * a.GY[mg]) + (nx * a.GX[og] + ny * a.GY[og]));
                    N1 = 0.5 * vm * ((nx * a.GX[mg + N2] + ny * a.GY[mg + N2]) +
                                     (nx * a.GX[og + N2] + ny * a.GY[og + N2]));
                }
                f0[pass] = -sc * a.c.geomFace * N0;
                f1[pass] = -sc * a.c.geomFace * N1;
                ms[pass] = sd[pass].y;
            }
        }
        __syncthreads();
        double lam = 0.0;
        if (active) {
            const int rb = el * N2 + eta * NGL, cb = el * N2 + xi;
            double d2 = 0, d3 = 0;
#pragma unroll
            for (int l = 0; l < NGL; ++l) {
                d2 += sDs[xi * NGL + l] * sF2[rb + l];
                d2 += sDs[eta * NGL + l] * sG2[cb + l * NGL];
                d3 += sDs[xi * NGL + l] * sF3[rb + l];
                d3 += sDs[eta * NGL + l] * sG3[cb + l * NGL];
            }
            const double J = a.Jinv[xid];
            double r0 = a.Qt[qid], r1 = a.Qt[qid + N2], r2 = a.Qt[qid + 2 * N2];
            r1 += J * d2;
            r2 += J * d3;
#pragma unroll
            for (int pass = 0; pass < 2; ++pass) {
                if (ms[pass] != 0) {
                    r1 += -ms[pass] * J * f0[pass];
                    r2 += -ms[pass] * J * f1[pass];
                }
            }
            const double h = a.q[qid], hu = a.q[qid + N2], hv = a.q[qid + 2 * N2];
            if (a.mode == 2) {
                a.Qt[qid] = r0; a.Qt[qid + N2] = r1; a.Qt[qid + 2 * N2] = r2;
            } else {
                const double dt = a.st[ins].dt;
                double q0, q1, q2;
                if (a.mode == 0) {
                    const double g0 = a.rkA * a.gRK[qid] + r0;
                    const double g1 = a.rkA * a.gRK[qid + N2] + r1;
                    const double g2 = a.rkA * a.gRK[qid + 2 * N2] + r2;
                    a.gRK[qid] = g0; a.gRK[qid + N2] = g1; a.gRK[qid + 2 * N2] = g2;
                    q0 = h + a.rkC * dt * g0;
                    q1 = hu + a.rkC * dt * g1;
                    q2 = hv + a.rkC * dt * g2;
                } else {
                    q0 = a.rkA * a.Qtmp[qid] + a.rkB * h + a.rkC * dt * r0;
                    q1 = a.rkA * a.Qtmp[qid + N2] + a.rkB * hu + a.rkC * dt * r1;
                    q2 = a.rkA * a.Qtmp[qid + 2 * N2] + a.rkB * hv + a.rkC * dt * r2;
                }
                a.q[qid] = q0; a.q[qid + N2] = q1; a.q[qid + 2 * N2] = q2;
                if (a.lam) lam = node_lambda(a.c, q0, q1, q2);
            }
            if (a.clear_act && nd == 0) a.act[e] = 0;  // read by no one until the next sensor pass
        }
        if (a.lam) warp_lambda<ElemShape<NGL>::THREADS>(lam, active, ins, a.st);
        __syncthreads();  // shared tiles are rewritten by the next iteration
    }
}

// BR1 gradient (lifted, h-scaled) of the elements of alist[0 .. *acount).
// okl/BR1_Gradient/calcGradient.okl:18-156, SurfaceKernelGradient.okl:16-150,
// scaleGradient.okl:17-60.
template <int NGL>
__global__ void __launch_bounds__(ElemShape<NGL>::THREADS) k_grad_list(ElemArgs a) {
    constexpr int N2 = NGL * NGL, NE = ElemShape<NGL>::NE;
    __shared__ double sDh[N2];
    __shared__ double su[NE * N2], sv[NE * N2];
    const int tid = threadIdx.x;
    const int el = tid / N2, nd = tid % N2;
    const int xi = nd % NGL, eta = nd / NGL;
    // the node's sides (-1: none) and its place along them
    const int sn[2] = {eta == 0 ? 0 : (eta == NGL - 1 ? 2 : -1), xi == NGL - 1 ? 1 : (xi == 0 ? 3 : -1)};
    const int jn[2] = {xi, eta};
    if (tid < N2) sDh[tid] = a.Dhat[tid];
    pdl_wait();
    const int count = *a.acount;
    for (int t = blockIdx.x; t * NE < count; t += gridDim.x) {
        if ((t + gridDim.x) * NE >= count) pdl_release();  // the CTA's last tile
        const int idx = t * NE + el;
        const bool inb = idx < count;
        const int e = inb ? a.alist[idx] : 0;
        const long xid = (long)e * N2 + nd, qid = (long)e * 3 * N2 + nd;
        const int s = el * N2 + nd;
        double h = 0;
        double fv[2][4];  // face values of the node's sides, loaded ahead of the barrier
        int ms[2] = {0, 0};
        if (inb) {
#pragma unroll
            for (int pass = 0; pass < 2; ++pass) {
                if (sn[pass] < 0) continue;
                const int4 sd = a.side[(long)e * 4 + sn[pass]];
                const int inc = sd.z ? jn[pass] : NGL - 1 - jn[pass];
                const double* ux = a.SGX + (long)sd.x * 2 * NGL + inc;
                const double* uy = a.SGY + (long)sd.x * 2 * NGL + inc;
                ms[pass] = sd.y;
                fv[pass][0] = ux[0]; fv[pass][1] = ux[NGL];
                fv[pass][2] = uy[0]; fv[pass][3] = uy[NGL];
            }
            h = a.q[qid];
            const double hu = a.q[qid + N2], hv = a.q[qid + 2 * N2];
            const double iv = (h > a.c.PosPresTOL) ? 1.0 / h : 0.0;
            su[s] = hu * iv; sv[s] = hv * iv;
        }
        __syncthreads();
        if (inb) {
            const int rb = el * N2 + eta * NGL, cb = el * N2 + xi;
            const double J = a.Jinv[xid];
            const double ye = a.Yeta[xid], yx = a.Yxi[xid], xe = a.Xeta[xid], xx = a.Xxi[xid];
            double gx0, gx1, gy0, gy1;
            {
                double uxi = 0, ueta = 0, vxi = 0, veta = 0;
#pragma unroll
                for (int l = 0; l < NGL; ++l) {
                    uxi += sDh[xi * NGL + l] * su[rb + l];
                    ueta += sDh[eta * NGL + l] * su[cb + l * NGL];
                    vxi += sDh[xi * NGL + l] * sv[rb + l];
                    veta += sDh[eta * NGL + l] * sv[cb + l * NGL];
                }
                const double ux = ye * uxi - yx * ueta, vx = ye * vxi - yx * veta;
                const double uy = -xe * uxi + xx * ueta, vy = -xe * vxi + xx * veta;
                gx0 = J * ux; gx1 = J * vx; gy0 = J * uy; gy1 = J * vy;
            }
#pragma unroll
            for (int pass = 0; pass < 2; ++pass) {
                if (ms[pass] != 0) {
                    if (pass == 0) gx0 += ms[pass] * fv[pass][0] * J;
                    else gx0 += ms[pass] * J * fv[pass][0];
                    gx1 += ms[pass] * J * fv[pass][1];
                    gy0 += ms[pass] * J * fv[pass][2];
                    gy1 += ms[pass] * J * fv[pass][3];
                }
            }
            const long gid = (long)e * 2 * N2 + nd;
            a.GX[gid] = h * gx0; a.GX[gid + N2] = h * gx1;
            a.GY[gid] = h * gy0; a.GY[gid + N2] = h * gy1;
        }
        __syncthreads();
    }
}

// Positivity limiter (okl/Positivity/PosPres.okl:17-223), optionally with the
// wave-speed maximum of the limited state.
//
// An element's means enter only where one of its depths is negative, so a
// block reads h, and the rest only where a node is shallow, an element has a
// negative depth or the wave speed is asked for: 8 instead of 32 B per node
// on wet elements.  Where the means are needed, every node forms its weight
// in parallel (the divisions) and one thread per sum adds them in the
// reference's order.
template <int NGL>
__global__ void __launch_bounds__(ElemShape<NGL>::THREADS) k_pospres(int K, const double* __restrict__ EleSizes,
                                                                   const double* __restrict__ GLw,
                                                                   const double* __restrict__ Jinv, double* q,
                                                                   const int* __restrict__ elem_inst, DevState* st,
                                                                   int lam_flag, PhysConst c) {
    constexpr int N2 = NGL * NGL, NE = ElemShape<NGL>::NE;
    __shared__ double sQ[NE * 3 * N2], sW[NE * N2];
    __shared__ double sAvg[NE][3];
    __shared__ int sNeg[NE];
    pdl_release();
    pdl_wait();
    const int tid = threadIdx.x;
    const int el = tid / N2, nd = tid % N2;
    const int e = blockIdx.x * NE + el;
    const bool inb = e < K;
    const int ins = inb ? inst_of(elem_inst, e) : 0;
    const bool active = inb && !st[ins].done;
    const long qid = (long)e * 3 * N2 + nd;
    double h = active ? q[qid] : 1.0, hu = 0.0, hv = 0.0;
    double lam = 0.0;
    const bool neg = h < 0.0;  // (NaN: no, as the reference's fmin passes it by)
    if (tid < NE) sNeg[tid] = 0;
    if (__syncthreads_or(neg)) {
        if (neg) sNeg[el] = 1;
        __syncthreads();
        const bool fix = active && sNeg[el];
        if (fix) {
            hu = q[qid + N2]; hv = q[qid + 2 * N2];
            double* s = sQ + el * 3 * N2 + nd;
            s[0] = h; s[N2] = hu; s[2 * N2] = hv;
            sW[el * N2 + nd] = GLw[nd % NGL] * GLw[nd / NGL] / Jinv[(long)e * N2 + nd];
        }
        __syncthreads();
        if (fix && nd < 3) {
            const double* s = sQ + el * 3 * N2 + nd * N2;
            double sum = 0.0;
            for (int l = 0; l < NGL; ++l)
                for (int k = 0; k < NGL; ++k) {
                    const int p = k * NGL + l;
                    sum += s[p] * sW[el * N2 + p];
                }
            sum = sum / EleSizes[e];
            if (nd == 0 && fabs(sum) < c.ZeroTOL) sum = 0.0;
            sAvg[el][nd] = sum;
        }
        __syncthreads();
        if (fix) {
            double hmin = 0.0;
            for (int k = 0; k < N2; ++k) hmin = fmin(hmin, sQ[el * 3 * N2 + k]);
            const double ha = sAvg[el][0], hua = sAvg[el][1], hva = sAvg[el][2];
            const double theta = (ha == hmin) ? 1.0 : fmin(1.0, ha / (ha - hmin));
            double hn = 0.0, hun = 0.0, hvn = 0.0;
            if (ha > 0.0) {
                hn = fabs(theta * (h - ha) + ha);
                if (hn > c.PosPresTOL) {
                    hun = theta * (hu - hua) + hua;
                    hvn = theta * (hv - hva) + hva;
                }
            }
            if (ha < 0.0) { hn = -1.0 / 0.0; hun = 0.0; hvn = 0.0; }  // -inf marks a failed limiter
            h = hn; hu = hun; hv = hvn;
            q[qid] = h; q[qid + N2] = hu; q[qid + 2 * N2] = hv;
            if (lam_flag) lam = node_lambda(c, h, hu, hv);
        }
    }
    if (active && !sNeg[el]) {
        if (h < c.PosPresTOL) {
            q[qid + N2] = 0.0; q[qid + 2 * N2] = 0.0;
            if (lam_flag) lam = node_lambda(c, h, 0.0, 0.0);
        } else if (lam_flag) {
            lam = node_lambda(c, h, q[qid + N2], q[qid + 2 * N2]);
        }
    }
    if (lam_flag) warp_lambda<ElemShape<NGL>::THREADS>(lam, active, ins, st);
}

// Wave-speed maximum of q (start of the time loop), all elements of one
// instance (that of element 0).  A resident grid strides over the nodes and
// each block ends with one atomic: with one per warp the atomics on the one
// key were the kernel (150 us at 6.55 million nodes; the loads take 24).
template <int NGL>
__global__ void __launch_bounds__(256) k_lambda(int K, const double* __restrict__ q,
                                                const int* __restrict__ elem_inst, DevState* st, PhysConst c) {
    constexpr int N2 = NGL * NGL;
    __shared__ unsigned long long s_key;
    if (threadIdx.x == 0) s_key = 0ull;
    __syncthreads();
    const long n = (long)K * N2;
    double lam = 0.0;
    for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
        const long e = i / N2, qid = e * 3 * N2 + (i - e * N2);
        const double v = node_lambda(c, q[qid], q[qid + N2], q[qid + 2 * N2]);
        lam = (isnan(v) || v > lam) ? v : lam;
    }
    const unsigned long long key = dbl_key(lam);
    const unsigned hi = (unsigned)(key >> 32), mhi = __reduce_max_sync(0xffffffffu, hi);
    const unsigned mlo = __reduce_max_sync(0xffffffffu, hi == mhi ? (unsigned)key : 0u);
    if ((threadIdx.x & 31) == 0) atomicMax(&s_key, ((unsigned long long)mhi << 32) | mlo);
    __syncthreads();
    if (threadIdx.x == 0) atomicMax(&st[inst_of(elem_inst, 0)].lam_key, s_key);
}

// Step bookkeeping per instance (src/deviceclass.cpp:897-930 and :1130):
// dt from the CFL and viscous limits, done flag when t >= T or the step cap
// is reached.
static __global__ void k_step_begin(int I, DevState* st, int ngl, int AV) {
    pdl_release();
    pdl_wait();
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= I) return;
    DevState& s = st[k];
    if (s.done) return;
    if (!(s.t < s.T) || (s.max_steps > 0 && s.steps >= s.max_steps)) { s.done = 1; return; }
    if (s.pause_on && s.steps > s.resume_steps && s.t >= s.pause_at) { s.done = 1; return; }
    const double lam = __longlong_as_double((long long)s.lam_key);
    if (s.lam_key == ~0ull || !isfinite(lam)) { s.status = ST_NONFINITE; s.done = 1; return; }
    const double dt_i = s.minEle / (double)ngl * s.CFL / lam;
    double dt;
    if (AV) {
        const double vmax = __longlong_as_double((long long)s.visc_key);
        const double dt_v = s.DFL / (pow((double)ngl, 2)) * pow(s.minEle, 2) / vmax;
        dt = fmin(s.T - s.t, fmin(dt_i, dt_v));
    } else {
        dt = fmin(s.T - s.t, dt_i);
    }
    s.dt = dt;
    s.lam_key = 0ull;
    s.visc_key = 0ull;
}

static __global__ void k_step_end(int I, DevState* st) {
    pdl_release();
    pdl_wait();
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= I) return;
    DevState& s = st[k];
    if (s.done) return;
    s.t += s.dt;
    s.steps += 1;
}

}  // namespace esdg
