// The time loop of a small single mesh as one kernel: every CTA keeps a
// contiguous range of elements -- q, the RK register and the metric terms
// -- in shared memory for the whole launch, and CTAs meet only through the
// traces of the faces between them.
//
// Why: on a mesh that fits the chip a stage's work takes a microsecond or
// two, while the step graph spends that on each of its 12 launches (their
// start-up, the drained last wave, the first loads of the next).  Here a
// stage is
//   the volume term of the first elements, while the neighbours' traces
//   arrive; the face fluxes of this CTA's sides into shared memory (a face
//   between two CTAs is evaluated by both, from the same operands);
//   lift, update, limiter, and on the last stage the wave-speed maximum; the
//   new traces that elements of other CTAs need go out with the update
//   (global memory, L2).
// There is no grid barrier: an exported value is one 16-byte word {value,
// epoch}, written and read as a single 128-bit access, and the reader polls
// the word itself until the epoch is this stage's.  That is one L2 round
// trip where a barrier needs a fence, an atomic and the reads after it.
// The words alternate between two buffers: a CTA writes stage k + 1's over
// stage k - 1's in its update of stage k, after it has read all its
// neighbours' words of stage k, which they wrote when they were done with
// stage k - 1.  The wave-speed
// maxima go round in the same way, once a step, one word per CTA.  Epochs
// grow from launch to launch, so no buffer is cleared.
// Every CTA takes the step's decisions (dt, end of the run) from the same
// numbers by the same arithmetic, as k_step_begin.
//
// The arithmetic per node and per face node is that of the step graph's
// kernels (pair_flux_raw, es_flux, the same update and limiter order), so
// the results are the same bits.
//
// Two CTAs per SM: one CTA's polls and barriers are covered by the other's
// arithmetic.  The block bound is 256 threads (128 registers, no spills)
// where those hold all of a CTA's nodes, else 384 (80 registers; spill stores
// and loads of 0 and 0 bytes at N = 1, 4 to 120 and 16 to 236 at N = 2..7): a
// second pass over the nodes costs more than the spills (51.8 against 59.6 us
// a step at 148,000 nodes of N = 4).  Where a CTA has
// threads to spare, whole warps take the face fluxes while the others run
// the volume term and gather the wave-speed words.
//
// Measured (B200, us per step, against the step graph): 15-17 against 37-40
// up to 25,000 nodes (bound by the latency of the exchange and of the FP64
// chains, not by work), 24-34 against 44-62 at 75,000, 46-56 against 62-88
// at 150,000, and equal to 1.25x faster at 240,000, about as much as the
// shared memory holds -- hence no other size limit.
//
// The launch is cooperative (all CTAs resident); every wait is bounded: a
// wait that runs out records ST_PEER_TIMEOUT and all CTAs leave (q and the
// step state keep what the launch started from).
#include "esdg_resident.hpp"

#include <algorithm>

#include "esdg_tma.cuh"

namespace esdg {

// Shared memory of a CTA with ne elements, T threads (doubles, then ints).
template <int NGL>
struct ResLayout {
    static constexpr int N2 = NGL * NGL;
    // q, RK register, seven metric terms and the side fluxes per element;
    // u, v, h^2 for one pass of ep elements; D
    __host__ __device__ static constexpr size_t doubles(int ne, int ep) {
        return (size_t)ne * (13 * N2 + 12 * NGL) + 3 * (size_t)ep * N2 + N2;
    }
    // face records (int4) and export flags (4 ne each); limiter: means (4 ne
    // doubles) and flags (ne); partial-dry treatment: flags (ne) and b
    __host__ __device__ static constexpr size_t bytes(int ne, int ep, bool extra, bool dry) {
        return 8 * (doubles(ne, ep) + (extra ? 4 * (size_t)ne : 0) + (dry ? (size_t)ne * N2 : 0)) +
               16 * 4 * (size_t)ne + 4 * (4 * (size_t)ne + (extra ? 2 * ne : 0)) + 32;
    }
};

struct ResCtl {
    double t, T, minEle, CFL, pause_at, dt_out;
    unsigned long long lam_out;
    int steps, max_steps, pause_on, resume_steps, done, done_out, status;
};

// One {value, epoch} word: a single 128-bit access each way (PTX ISA 8.3,
// ld/st.b128), so a reader never sees half of one.
struct __align__(16) ResWord {
    unsigned long long v, epoch;
};
__device__ __forceinline__ void res_put(ResWord* p, unsigned long long v, unsigned long long epoch) {
    asm volatile("{\n\t.reg .b128 w;\n\tmov.b128 w, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], w;\n\t}" ::"l"(p),
                 "l"(v), "l"(epoch)
                 : "memory");
}
__device__ __forceinline__ ResWord res_get(const ResWord* p) {
    ResWord w;
    asm volatile("{\n\t.reg .b128 w;\n\tld.relaxed.gpu.global.b128 w, [%2];\n\tmov.b128 {%0, %1}, w;\n\t}"
                 : "=l"(w.v), "=l"(w.epoch)
                 : "l"(p)
                 : "memory");
    return w;
}
// Waits for three words (stride apart) of this epoch.
__device__ __forceinline__ bool res_poll3(const ResWord* p, int stride, unsigned long long epoch, long long limit,
                                          double& a, double& b, double& c) {
    const long long lim = limit > 0 ? limit : 4000000000ll;
    long long t0 = 0;
    for (;;) {
        const ResWord x = res_get(p), y = res_get(p + stride), z = res_get(p + 2 * stride);
        a = __longlong_as_double((long long)x.v);
        b = __longlong_as_double((long long)y.v);
        c = __longlong_as_double((long long)z.v);
        if (x.epoch == epoch && y.epoch == epoch && z.epoch == epoch) return true;
        const long long now = clock64();
        if (t0 == 0) t0 = now;
        else if (now - t0 > lim) return false;
    }
}
__device__ __forceinline__ bool res_poll(const ResWord* p, unsigned long long epoch, long long limit,
                                         unsigned long long& v) {
    const long long lim = limit > 0 ? limit : 4000000000ll;
    long long t0 = 0;
    for (;;) {
        const ResWord x = res_get(p);
        v = x.v;
        if (x.epoch == epoch) return true;
        const long long now = clock64();
        if (t0 == 0) t0 = now;
        else if (now - t0 > lim) return false;
    }
}

// Maximum of a key over the warp (all lanes).
__device__ __forceinline__ unsigned long long res_warp_max(unsigned long long key) {
    const unsigned hi = (unsigned)(key >> 32);
    const unsigned mhi = __reduce_max_sync(0xffffffffu, hi);
    const unsigned mlo = __reduce_max_sync(0xffffffffu, hi == mhi ? (unsigned)key : 0u);
    return ((unsigned long long)mhi << 32) | mlo;
}

template <int NGL, bool EXTRA, int THREADS>
__global__ void __launch_bounds__(THREADS, 2) k_resident(const ResArgs a) {
    constexpr int N2 = NGL * NGL;
    // The exported words go out with the update where a thread's registers
    // have room for it (the small block: 18.9 -> 16.4 us a step at 256
    // elements of N = 3), else from the finished state at the next stage's
    // start (the large block spills for it: 5 % slower at 75,000 nodes), and
    // behind the limiter.
    constexpr bool EARLY = THREADS == 256 && !EXTRA;
    extern __shared__ __align__(16) double rsm[];
    __shared__ ResCtl ctl;
    __shared__ unsigned long long s_lam, s_key[2];
    __shared__ int s_nf, s_nx, s_bad;
    const int tid = threadIdx.x, T = blockDim.x;
    const int EP = a.ep;
    const int e0 = blockIdx.x * a.ne;
    const int ne = min(a.ne, a.K - e0);
    int4* sface = reinterpret_cast<int4*>(rsm);  // faces of this CTA: face, left, right element, sides and flags
    double* sq = rsm + 8 * (size_t)a.ne;    // [ne][3][N2]
    double* sg = sq + (size_t)a.ne * 3 * N2;
    double* sJ = sg + (size_t)a.ne * 3 * N2;
    double* sBx = sJ + (size_t)a.ne * N2;
    double* sBy = sBx + (size_t)a.ne * N2;
    double* sYx = sBy + (size_t)a.ne * N2;
    double* sYe = sYx + (size_t)a.ne * N2;
    double* sXx = sYe + (size_t)a.ne * N2;
    double* sXe = sXx + (size_t)a.ne * N2;
    double* sF = sXe + (size_t)a.ne * N2;   // [ne][4][3][NGL]
    double* su = sF + (size_t)a.ne * 12 * NGL;
    double* sv = su + EP * N2;
    double* sh2 = sv + EP * N2;
    double* sD = sh2 + EP * N2;
    double* sAvg = sD + N2;                 // [ne][4] (EXTRA)
    // exported sides: flags [ne][4] (EARLY), else a list
    double* sB = sAvg + (EXTRA ? 4 * (size_t)a.ne : 0);  // [ne][N2] b (partial-dry treatment)
    int* sexp = reinterpret_cast<int*>(sB + (EXTRA && a.dry_on ? (size_t)a.ne * N2 : 0));
    int* sneg = sexp + 4 * a.ne;             // [ne] element has a negative depth (EXTRA)
    int* sdry = sneg + a.ne;                 // [ne] element has a node below PosPresTOL (EXTRA)

    if (tid == 0) {
        s_nf = 0;
        s_nx = 0;
        s_lam = 0ull;
        s_bad = 0;
        s_key[0] = a.st->lam_key;
        s_key[1] = 0ull;
        const DevState& S = *a.st;
        ctl.t = S.t; ctl.T = S.T; ctl.minEle = S.minEle; ctl.CFL = S.CFL; ctl.pause_at = S.pause_at;
        ctl.dt_out = S.dt;
        ctl.lam_out = S.lam_key;
        ctl.steps = S.steps; ctl.max_steps = S.max_steps; ctl.pause_on = S.pause_on;
        ctl.resume_steps = S.resume_steps; ctl.done = S.done; ctl.done_out = S.done; ctl.status = ST_OK;
    }
    for (int i = tid; i < ne * 3 * N2; i += T) {
        sq[i] = a.q[(size_t)e0 * 3 * N2 + i];
        if (!a.ssp) sg[i] = a.gRK[(size_t)e0 * 3 * N2 + i];
    }
    for (int i = tid; i < ne * N2; i += T) {
        const size_t k = (size_t)e0 * N2 + i;
        sJ[i] = a.Jinv[k]; sBx[i] = a.Bx[k]; sBy[i] = a.By[k];
        sYx[i] = a.Yxi[k]; sYe[i] = a.Yeta[k]; sXx[i] = a.Xxi[k]; sXe[i] = a.Xeta[k];
    }
    for (int i = tid; i < N2; i += T) sD[i] = a.D[i];
    if (EXTRA && a.dry_on) {
        for (int i = tid; i < ne * N2; i += T) sB[i] = a.B[(size_t)e0 * N2 + i];
        for (int i = tid; i < ne; i += T) sdry[i] = 0;
    }
    __syncthreads();
    // Faces to evaluate: those whose master side is here, and those whose
    // slave side is here with the master in another CTA (evaluated there
    // too).  Sides whose neighbour is in another CTA export their trace.
    for (int i = tid; i < 4 * ne; i += T) {
        const int e = e0 + i / 4, sd = i % 4;
        const int f = a.side[(size_t)e * 4 + sd].x;
        const int4 t = a.ftab[f];
        const bool master = t.x == e && (t.z & 3) == sd;
        const int other = master ? t.y : t.x;
        const bool local = other >= e0 && other < e0 + ne;
        if (master || !local) sface[atomicAdd(&s_nf, 1)] = make_int4(f, t.x, t.y, (t.z & 31) | (t.w << 8));
        const bool out = other >= 0 && !local;
        if (EARLY) sexp[i] = out;
        else if (out) sexp[atomicAdd(&s_nx, 1)] = i;
    }
    __syncthreads();
    const int nfaces = s_nf;
    const int npass = (ne + EP - 1) / EP;
    const int el0 = tid / N2, nd = tid % N2;
    const int xi = nd % NGL, eta = nd / NGL;
    const bool worker = el0 < EP;
    // threads of the face fluxes: the warps from fbase on, or all (fbase = 0)
    const int fbase = a.fbase;
    const int ft = tid - fbase, fn = T - fbase;
    const double g = a.c.g;
    unsigned long long epoch = a.epoch;  // grows by one a stage
    int ran = 0;                         // steps of this launch
    double dt = 0.0;
    const size_t half = (size_t)a.K * 12 * NGL;
    ResWord* lamw = a.lam;               // [2][gridDim.x]

    // volume term of node nd of local element el, scratch slot el0
    auto volume = [&](int el, double& r0, double& r1, double& r2) {
        const double* q = sq + el * 3 * N2;
        const int m = el * N2, z = el0 * N2;
        const double h = q[nd], hu = q[nd + N2], hv = q[nd + 2 * N2];
        const double uL = su[z + nd], vL = sv[z + nd], h2L = sh2[z + nd];
        const double ye = sYe[m + nd], yx = sYx[m + nd], xe = sXe[m + nd], xx = sXx[m + nd];
        double d1 = 0.0, d2 = 0.0, d3 = 0.0;
#pragma unroll
        for (int l = 0; l < NGL; ++l) {
            const int p = eta * NGL + l;
            const double dl = sD[xi * NGL + l];
            double f1, f2, f3;
            pair_flux_raw<false>(g, h, hu, hv, uL, vL, h2L, ye, xe, q[p], q[p + N2], q[p + 2 * N2], su[z + p],
                                 sv[z + p], sh2[z + p], sYe[m + p], sXe[m + p], f1, f2, f3);
            d1 += dl * f1; d2 += dl * f2; d3 += dl * f3;
        }
#pragma unroll
        for (int l = 0; l < NGL; ++l) {
            const int p = xi + l * NGL;
            const double dl = sD[eta * NGL + l];
            double f1, f2, f3;
            pair_flux_raw<true>(g, h, hu, hv, uL, vL, h2L, yx, xx, q[p], q[p + N2], q[p + 2 * N2], su[z + p],
                                sv[z + p], sh2[z + p], sYx[m + p], sXx[m + p], f1, f2, f3);
            d1 += dl * f1; d2 += dl * f2; d3 += dl * f3;
        }
        d1 *= 0.25;
        d2 *= 0.125;
        d3 *= 0.125;
        const double J = sJ[m + nd];
        r0 = -J * d1;
        r1 = -J * d2 - g * h * sBx[m + nd];
        r2 = -J * d3 - g * h * sBy[m + nd];
        if (EXTRA && a.dry_on && sdry[el])
            pd_volume<NGL>(a.c, a.Dc, a.Dup, a.Ddn, q, sB + el * N2, eta, xi, ye, yx, xe, xx, J, r1, r2);
    };
    auto scratch = [&](int el) {
        const double* q = sq + el * 3 * N2;
        const double h = q[nd];
        const double ih = (h > 0) ? 1.0 / h : 0.0;
        su[el0 * N2 + nd] = q[nd + N2] * ih;
        sv[el0 * N2 + nd] = q[nd + 2 * N2] * ih;
        sh2[el0 * N2 + nd] = h * h;
        // FindDryElements: min(1, h) < PosPresTOL (NaN passes by)
        if (EXTRA && a.dry_on && (h < a.c.PosPresTOL || 1.0 < a.c.PosPresTOL)) sdry[el] = 1;
    };
    double lam = 0.0;   // this thread's wave-speed maximum of the step (NaN sticks)
    auto fold = [&](double v) { lam = (isnan(v) || v > lam) ? v : lam; };
    // lift (sides 0/2, then 1/3) and update of node nd of local element el
    auto finish = [&](int el, double r0, double r1, double r2, double A, double Bc, double C, bool first, bool last) {
        const int m = el * N2 + nd;
        double* q = sq + el * 3 * N2 + nd;
        double* gk = sg + el * 3 * N2 + nd;
        const double J = sJ[m];
        const double db = 0.0;
#pragma unroll
        for (int pass = 0; pass < 2; ++pass) {
            int sd = -1, j = 0;
            if (pass == 0) {
                if (eta == 0) { sd = 0; j = xi; }
                else if (eta == NGL - 1) { sd = 2; j = xi; }
            } else {
                if (xi == NGL - 1) { sd = 1; j = eta; }
                else if (xi == 0) { sd = 3; j = eta; }
            }
            if (sd >= 0) {
                const double* fp = sF + (el * 4 + sd) * 3 * NGL + j;
                r0 += fp[0] * J;
                r1 += J * fp[NGL] + J * db;
                r2 += J * fp[2 * NGL] + J * db;
            }
        }
        const double h = q[0], hu = q[N2], hv = q[2 * N2];
        if (EXTRA && a.dry_on && nd == 0) sdry[el] = 0;  // read by this pass's volume terms, behind a barrier
        double q0, q1, q2;
        if (!a.ssp) {
            const double g0 = A * gk[0] + r0, g1 = A * gk[N2] + r1, g2 = A * gk[2 * N2] + r2;
            gk[0] = g0; gk[N2] = g1; gk[2 * N2] = g2;
            q0 = h + C * dt * g0;
            q1 = hu + C * dt * g1;
            q2 = hv + C * dt * g2;
        } else {
            if (first) { gk[0] = h; gk[N2] = hu; gk[2 * N2] = hv; }  // the step's start state
            q0 = A * gk[0] + Bc * h + C * dt * r0;
            q1 = A * gk[N2] + Bc * hu + C * dt * r1;
            q2 = A * gk[2 * N2] + Bc * hv + C * dt * r2;
        }
        q[0] = q0; q[N2] = q1; q[2 * N2] = q2;
        if (EXTRA && a.PP) {
            if (q0 < 0.0) sneg[el] = 1;
        } else if (last) {
            fold(node_lambda(a.c, q0, q1, q2));
        }
        if (EARLY) {
            // the next stage's words, as soon as the values are there
            ResWord* tr = a.tr + ((epoch + 1) & 1) * half;
#pragma unroll
            for (int pass = 0; pass < 2; ++pass) {
                const int sd = pass == 0 ? (eta == 0 ? 0 : (eta == NGL - 1 ? 2 : -1)) : (xi == NGL - 1 ? 1 : (xi == 0 ? 3 : -1));
                if (sd >= 0 && sexp[el * 4 + sd]) {
                    ResWord* o = tr + ((size_t)(e0 + el) * 4 + sd) * 3 * NGL + (pass == 0 ? xi : eta);
                    res_put(o, (unsigned long long)__double_as_longlong(q0), epoch + 1);
                    res_put(o + NGL, (unsigned long long)__double_as_longlong(q1), epoch + 1);
                    res_put(o + 2 * NGL, (unsigned long long)__double_as_longlong(q2), epoch + 1);
                }
            }
        }
    };
    // words of every exported side for stage ep
    auto export_all = [&](unsigned long long ep) {
        ResWord* tr = a.tr + (ep & 1) * half;
        const int n = (EARLY ? 4 * ne : s_nx) * NGL;
        for (int i = tid; i < n; i += T) {
            const int j = i % NGL, k = EARLY ? i / NGL : sexp[i / NGL];
            if (EARLY && !sexp[k]) continue;
            const double* q = sq + (k / 4) * 3 * N2 + trace_offset(k & 3, j, NGL);
            ResWord* o = tr + ((size_t)(e0 + k / 4) * 4 + (k & 3)) * 3 * NGL + j;
            res_put(o, (unsigned long long)__double_as_longlong(q[0]), ep);
            res_put(o + NGL, (unsigned long long)__double_as_longlong(q[N2]), ep);
            res_put(o + 2 * NGL, (unsigned long long)__double_as_longlong(q[2 * N2]), ep);
        }
    };
    if (EARLY) export_all(epoch + 1);

    bool leave = false;
    while (!leave) {
        for (int s = 0; s < a.stages; ++s) {
            const bool last = s == a.stages - 1;
            ++epoch;
            const ResWord* tr = a.tr + (epoch & 1) * half;
            if (!EARLY) export_all(epoch);
            if (s == 0 && tid == 0) {
                if (ran > 0) res_put(lamw + (ran & 1) * gridDim.x + blockIdx.x, s_lam, epoch);
                s_lam = 0ull;
            }
            if (worker && el0 < ne) scratch(el0);
            if (EXTRA && a.PP)
                for (int i = tid; i < ne; i += T) sneg[i] = 0;
            if (fbase == 0) __syncthreads();
            else if (ft < 0) asm volatile("bar.sync 1, %0;" ::"r"(fbase) : "memory");  // the node warps' scratch
            double r0 = 0.0, r1 = 0.0, r2 = 0.0;
            if (worker && el0 < ne) volume(el0, r0, r1, r2);
            // ---- face fluxes of this CTA's sides ----
            bool ok = true;
            for (int i = ft; i >= 0 && i < nfaces * NGL; i += fn) {
                const int4 t = sface[i / NGL];
                const int j = i % NGL, f = t.x, eL = t.y, eR = t.z;
                const long ex = (long)f * NGL + j;
                const int sL = t.w & 3, sR = (t.w >> 2) & 3, same = (t.w >> 4) & 1, w = t.w >> 8;
                const double nx = a.nx[ex], ny = a.ny[ex], sc = a.scal[ex], bLx = a.bL[ex];
                const int ir = same ? j : NGL - 1 - j;
                const double bRx = a.bR[(long)f * NGL + ir];
                const bool locL = eL >= e0 && eL < e0 + ne, locR = eR >= e0 && eR < e0 + ne;
                auto trace = [&](int e, bool loc, int sd, int k, double& h, double& hu, double& hv) {
                    if (loc) {
                        const double* q = sq + (e - e0) * 3 * N2 + trace_offset(sd, k, NGL);
                        h = q[0]; hu = q[N2]; hv = q[2 * N2];
                    } else {
                        h = hu = hv = 0.0;
                        ok = ok && res_poll3(tr + ((size_t)e * 4 + sd) * 3 * NGL + k, NGL, epoch, a.wait_limit, h, hu,
                                             hv);
                    }
                };
                double hL, huL, hvL, hR, huR, hvR;
                trace(eL, locL, sL, j, hL, huL, hvL);
                if (eR >= 0) {
                    trace(eR, locR, sR, ir, hR, huR, hvR);
                } else {
                    const long exr = (long)f * NGL + ir;
                    double h, hu, hv;
                    trace(eL, locL, sL, ir, h, hu, hv);
                    wall_ghost(a.nx[exr], a.ny[exr], h, hu, hv, hR, huR, hvR);
                }
                double F0, F1, F2;
                if (a.numflux == 0) es_flux<0>(a.c, nx, ny, hL, huL, hvL, hR, huR, hvR, bLx, bRx, F0, F1, F2);
                else if (a.numflux == 2) es_flux<2>(a.c, nx, ny, hL, huL, hvL, hR, huR, hvR, bLx, bRx, F0, F1, F2);
                else es_flux<3>(a.c, nx, ny, hL, huL, hvL, hR, huR, hvR, bLx, bRx, F0, F1, F2);
                const double v0 = sc * a.c.geomFace * F0, v1 = sc * a.c.geomFace * F1, v2 = sc * a.c.geomFace * F2;
                if (locL) {
                    double* o = sF + ((eL - e0) * 4 + sL) * 3 * NGL + ((w & 1) ? j : NGL - 1 - j);
                    const bool n = (w & 2) != 0;
                    o[0] = n ? v0 : -v0; o[NGL] = n ? v1 : -v1; o[2 * NGL] = n ? v2 : -v2;
                }
                if (locR) {
                    double* o = sF + ((eR - e0) * 4 + sR) * 3 * NGL + ((w & 4) ? j : NGL - 1 - j);
                    const bool n = (w & 8) != 0;
                    o[0] = n ? v0 : -v0; o[NGL] = n ? v1 : -v1; o[2 * NGL] = n ? v2 : -v2;
                }
            }
            if (s == 0 && ran > 0 && (fbase == 0 || ft < 0)) {
                // the wave-speed keys of all CTAs, by whole warps that have
                // no face fluxes to form (or all); a thread's words are
                // requested together, the late ones again
                const ResWord* lw = lamw + (ran & 1) * gridDim.x;
                const int gn = fbase == 0 ? T : fbase;
                unsigned long long key = 0ull;
                if constexpr (THREADS == 256) {
                    for (int i0 = tid; i0 < (int)gridDim.x; i0 += 4 * gn) {
                        ResWord x[4];
#pragma unroll
                        for (int k = 0; k < 4; ++k)
                            if (i0 + k * gn < (int)gridDim.x) x[k] = res_get(lw + i0 + k * gn);
#pragma unroll
                        for (int k = 0; k < 4; ++k)
                            if (i0 + k * gn < (int)gridDim.x) {
                                unsigned long long v = x[k].v;
                                if (x[k].epoch != epoch) ok = ok && res_poll(lw + i0 + k * gn, epoch, a.wait_limit, v);
                                key = v > key ? v : key;
                            }
                    }
                } else {
                    for (int i = tid; i < (int)gridDim.x; i += gn) {
                        unsigned long long v = 0ull;
                        ok = ok && res_poll(lw + i, epoch, a.wait_limit, v);
                        key = v > key ? v : key;
                    }
                }
                key = res_warp_max(key);
                if ((tid & 31) == 0) atomicMax(&s_key[ran & 1], key);
            }
            if (!ok) s_bad = 1;
            __syncthreads();
            if (s_bad) {  // a wait ran out: this CTA leaves, the others' waits run out too
                if (tid == 0) atomicExch(&a.st->status, ST_PEER_TIMEOUT);
                return;
            }
            if (s == 0) {
                // the step's start (k_step_begin), the same in every thread
                const unsigned long long key = s_key[ran & 1];
                const double l = __longlong_as_double((long long)key);
                int done = ctl.done, status = ST_OK;
                if (ran >= a.nsteps || done) leave = true;
                else if (!(ctl.t < ctl.T) || (ctl.max_steps > 0 && ctl.steps >= ctl.max_steps)) done = 1;
                else if (ctl.pause_on && ctl.steps > ctl.resume_steps && ctl.t >= ctl.pause_at) done = 1;
                else if (key == ~0ull || !isfinite(l)) { status = ST_NONFINITE; done = 1; }
                else {
                    const double dt_i = ctl.minEle / (double)NGL * ctl.CFL / l;
                    dt = fmin(ctl.T - ctl.t, dt_i);
                }
                if (tid == 0) {
                    s_key[(ran + 1) & 1] = 0ull;
                    ctl.lam_out = key;
                    ctl.done_out = done;
                    ctl.status = status;
                    if (!done && !leave) ctl.dt_out = dt;
                }
                if (done) leave = true;
                if (leave) break;
            }
            // ---- lift and update, pass by pass ----
            const double A = a.rkA[s], Bc = a.rkB[s], C = a.rkC[s];
            if (worker && el0 < ne) finish(el0, r0, r1, r2, A, Bc, C, s == 0, last);
            for (int p = 1; p < npass; ++p) {
                const int el = p * EP + el0;
                const bool on = worker && el < ne;
                __syncthreads();  // the scratch of the pass before is free
                if (on) scratch(el);
                __syncthreads();
                if (on) volume(el, r0, r1, r2);
                __syncthreads();  // every node's pairs are done before the first node is updated
                if (on) finish(el, r0, r1, r2, A, Bc, C, s == 0, last);
            }
            if (EXTRA && a.PP) {
                // Positivity limiter (k_pospres, the same sums in the same
                // order); the means are needed only where a depth is negative.
                __syncthreads();
                for (int el = tid; el < ne; el += T) {
                    if (!sneg[el]) continue;
                    const double* q = sq + el * 3 * N2;
                    double hmin = 0.0, ha = 0.0, hua = 0.0, hva = 0.0;
                    for (int l = 0; l < NGL; ++l)
                        for (int k = 0; k < NGL; ++k) {
                            const int p = k * NGL + l;
                            const double w = a.GLw[l] * a.GLw[k] / sJ[el * N2 + p];
                            ha += q[p] * w;
                            hua += q[p + N2] * w;
                            hva += q[p + 2 * N2] * w;
                            hmin = fmin(hmin, q[p]);
                        }
                    const double es = a.EleSizes[e0 + el];
                    ha = ha / es;
                    if (fabs(ha) < a.c.ZeroTOL) ha = 0.0;
                    sAvg[el * 4] = ha;
                    sAvg[el * 4 + 1] = hua / es;
                    sAvg[el * 4 + 2] = hva / es;
                    sAvg[el * 4 + 3] = hmin;
                }
                __syncthreads();
                for (int i = tid; i < ne * N2; i += T) {
                    const int el = i / N2;
                    double* q = sq + el * 3 * N2 + (i - el * N2);
                    double h = q[0], hu = q[N2], hv = q[2 * N2];
                    if (sneg[el]) {
                        const double ha = sAvg[el * 4], hua = sAvg[el * 4 + 1], hva = sAvg[el * 4 + 2];
                        const double hmin = sAvg[el * 4 + 3];
                        const double theta = (ha == hmin) ? 1.0 : fmin(1.0, ha / (ha - hmin));
                        double hn = 0.0, hun = 0.0, hvn = 0.0;
                        if (ha > 0.0) {
                            hn = fabs(theta * (h - ha) + ha);
                            if (hn > a.c.PosPresTOL) {
                                hun = theta * (hu - hua) + hua;
                                hvn = theta * (hv - hva) + hva;
                            }
                        }
                        if (ha < 0.0) { hn = -1.0 / 0.0; hun = 0.0; hvn = 0.0; }
                        h = hn; hu = hun; hv = hvn;
                        q[0] = h; q[N2] = hu; q[2 * N2] = hv;
                    } else if (h < a.c.PosPresTOL) {
                        hu = 0.0; hv = 0.0;
                        q[N2] = 0.0; q[2 * N2] = 0.0;
                    }
                    if (last) fold(node_lambda(a.c, h, hu, hv));
                }
            }
            if (last) {
                // the step's wave-speed key of this CTA (a maximum: any order)
                const unsigned long long key = res_warp_max(dbl_key(lam));
                lam = 0.0;
                if ((tid & 31) == 0) atomicMax(&s_lam, key);
                if (tid == 0) {  // the step's end (k_step_end)
                    ctl.t += dt;
                    ctl.steps += 1;
                }
            }
            __syncthreads();
        }
        if (!leave) ++ran;
    }
    for (int i = tid; i < ne * 3 * N2; i += T) {
        a.q[(size_t)e0 * 3 * N2 + i] = sq[i];
        if (!a.ssp) a.gRK[(size_t)e0 * 3 * N2 + i] = sg[i];
    }
    // Every CTA has read the state this launch started from: CTA 0 leaves
    // at a step's start, after words of this launch from all its neighbours,
    // and for ran > 0 from all CTAs; a launch that leaves at its first step
    // changes nothing that the others decide by (done_out follows from the
    // same numbers, and they test it first).
    if (blockIdx.x == 0 && tid == 0) {
        DevState& S = *a.st;
        S.done = ctl.done_out;
        if (ctl.status != ST_OK) S.status = ctl.status;
        if (ran > 0) {
            S.t = ctl.t;
            S.dt = ctl.dt_out;
            S.steps = ctl.steps;
            S.lam_key = ctl.lam_out;
            S.visc_key = 0ull;
        }
    }
}

// Dynamic shared memory of a CTA at most: two CTAs an SM.
constexpr size_t RES_SMEM = (size_t)112 * 1024;

template <int NGL>
static ResShape shape_of(int K, int sms, bool extra, bool dry) {
    constexpr int N2 = NGL * NGL;
    ResShape s{0, 0, 0, 0, 0, 0, 0};
    const int ne = (K + 2 * sms - 1) / (2 * sms);
    // the small block where its threads hold all nodes, else the large one,
    // in passes of equal size
    s.block = ne * N2 <= 256 ? 256 : 384;
    const int npass = (ne + s.block / N2 - 1) / (s.block / N2);
    s.ep = (ne + npass - 1) / npass;
    s.smem = ResLayout<NGL>::bytes(ne, s.ep, extra, dry);
    if (s.smem > RES_SMEM) return s;
    // whole warps for the face nodes (at most four sides an element) where
    // all of them fit beside the nodes; else every thread does both
    const int nodes = (s.ep * N2 + 31) / 32 * 32, faces = (4 * ne * NGL + 31) / 32 * 32;
    const bool split = npass == 1 && nodes + faces <= s.block;
    s.fbase = split ? nodes : 0;
    s.threads = split ? nodes + faces : std::min(s.block, std::max(nodes, faces));
    s.ne = ne;
    s.grid = (K + ne - 1) / ne;
    return s;
}

#define ESDG_RES_DISPATCH(ngl, F)   \
    switch (ngl) {                  \
        case 2: F(2); break;        \
        case 3: F(3); break;        \
        case 4: F(4); break;        \
        case 5: F(5); break;        \
        case 6: F(6); break;        \
        case 7: F(7); break;        \
        case 8: F(8); break;        \
        default: break;             \
    }

ResShape resident_shape(int ngl, int K, int sms, bool extra, bool dry) {
    ResShape s{0, 0, 0, 0, 0, 0, 0};
#define ESDG_F(n) s = shape_of<n>(K, sms, extra, dry)
    ESDG_RES_DISPATCH(ngl, ESDG_F)
#undef ESDG_F
    return s;
}

template <int NGL>
static const void* kernel_of(int block, bool extra) {
    if (block == 256) return extra ? (const void*)k_resident<NGL, true, 256> : (const void*)k_resident<NGL, false, 256>;
    return extra ? (const void*)k_resident<NGL, true, 384> : (const void*)k_resident<NGL, false, 384>;
}

static const void* kernel_of(int ngl, const ResShape& s, bool extra) {
    const void* k = nullptr;
#define ESDG_F(n) k = kernel_of<n>(s.block, extra)
    ESDG_RES_DISPATCH(ngl, ESDG_F)
#undef ESDG_F
    return k;
}

// The attribute belongs to the function, not to a solver: always the bound,
// whatever this mesh needs, or a smaller solver of the same instance would
// take it from a larger one.
cudaError_t resident_setup(int ngl, const ResShape& s, bool extra) {
    return cudaFuncSetAttribute(kernel_of(ngl, s, extra), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)RES_SMEM);
}

cudaError_t resident_launch(const ResArgs& a, const ResShape& s, bool extra, cudaStream_t stream) {
    ResArgs args = a;
    args.ne = s.ne;
    args.ep = s.ep;
    args.fbase = s.fbase;
    void* p[] = {&args};
    return cudaLaunchCooperativeKernel(kernel_of(a.ngl, s, extra), dim3(s.grid), dim3(s.threads), p, s.smem, stream);
}

}  // namespace esdg
