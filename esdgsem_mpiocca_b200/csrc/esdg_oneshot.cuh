// Element kernel without a pipeline: one block per NE elements, one thread
// per node, every operand read by the thread that uses it.  The same
// arithmetic per node as k_element_tma (every operation in the same order, so
// the same bits).
//
// Where it is the faster one: degrees whose elements fill the pipelined
// kernels' tiles badly (N = 6: 49 nodes, four elements a tile are 196 of 224
// lanes, and two per thread 98 of 128) on meshes that stay in L2, where
// there is no HBM latency for a pipeline to hide; viscous meshes of N = 1; and
// small meshes with little more than one tile per resident CTA (rule_variant
// has the times).
#pragma once

#include "esdg_tma.cuh"

namespace esdg {

constexpr int ONESHOT_VARIANTS = 1;

// GEN as for k_element_tma.
template <int NGL, int GEN = 1>
__global__ void __launch_bounds__(ElemShape<NGL>::THREADS) k_element_oneshot(ElemArgs a) {
    constexpr int N2 = NGL * NGL, NE = ElemShape<NGL>::NE, ND = NE * N2;
    __shared__ double sD[N2];
    __shared__ double sh[ND], shu[ND], shv[ND], su[ND], sv[ND], sh2[ND];
    __shared__ double sYe[ND], sYx[ND], sXe[ND], sXx[ND];
    const int tid = threadIdx.x;
    const int el = tid / N2, nd = tid % N2;
    const int e0 = blockIdx.x * NE;
    const int xi = nd % NGL, eta = nd / NGL;
    if (tid < N2) sD[tid] = a.D[tid];
    pdl_release();
    pdl_wait();
    if (GEN != 0 && a.extent && e0 >= a.extent[0]) return;  // whole block past the live extent
    const int e = e0 + el;
    const bool inb = e < a.K;
    const int ins = (GEN != 0 && inb) ? inst_of(a.elem_inst, e) : 0;
    const bool active = inb && !a.st[ins].done;
    const bool to_list = GEN != 0 && active && a.act && a.act[e] != 0;
    if (GEN != 0 && a.act && tid < 32) list_tile(a, e0, NE);
    const long xid = (long)e * N2 + nd, qid = (long)e * 3 * N2 + nd;
    const int s = el * N2 + nd;
    // every global read of this thread ahead of the barrier: state and
    // metrics (staged for the partners), Jinv, Bx, By, the second register
    // and the face fluxes of the node's sides
    double h = 0, hu = 0, hv = 0, J = 0, bx = 0, by = 0, o0 = 0, o1 = 0, o2 = 0, dt = 0;
    double f[2][3];
    bool has[2] = {false, false};
    if (active) {
        h = a.q[qid]; hu = a.q[qid + N2]; hv = a.q[qid + 2 * N2];
        sYe[s] = a.Yeta[xid]; sYx[s] = a.Yxi[xid]; sXe[s] = a.Xeta[xid]; sXx[s] = a.Xxi[xid];
        J = a.Jinv[xid]; bx = a.Bx[xid]; by = a.By[xid];
        if (a.mode == 0) { o0 = a.gRK[qid]; o1 = a.gRK[qid + N2]; o2 = a.gRK[qid + 2 * N2]; }
        else if (a.mode == 1) { o0 = a.Qtmp[qid]; o1 = a.Qtmp[qid + N2]; o2 = a.Qtmp[qid + 2 * N2]; }
        if (a.mode != 2) dt = a.st[ins].dt;
#pragma unroll
        for (int pass = 0; pass < 2; ++pass) {
            int side = -1, j = 0;
            if (pass == 0) {
                if (eta == 0) { side = 0; j = xi; }
                else if (eta == NGL - 1) { side = 2; j = xi; }
            } else {
                if (xi == NGL - 1) { side = 1; j = eta; }
                else if (xi == 0) { side = 3; j = eta; }
            }
            if (side >= 0) {
                has[pass] = true;
                const double* fp = a.SP + side_flux_at(e, side, 0, j, NGL);
                f[pass][0] = fp[0]; f[pass][1] = fp[NGL]; f[pass][2] = fp[2 * NGL];
            }
        }
        sh[s] = h; shu[s] = hu; shv[s] = hv;
        const double ih = (h > 0) ? 1.0 / h : 0.0;
        su[s] = hu * ih;
        sv[s] = hv * ih;
        sh2[s] = h * h;
    }
    __syncthreads();
    double lam = 0.0;
    if (active) {
        const int rb = el * N2 + eta * NGL, cb = el * N2 + xi;
        const double g = a.c.g, uL = su[s], vL = sv[s], h2L = sh2[s];
        const double ye = sYe[s], yx = sYx[s], xe = sXe[s], xx = sXx[s];
        double d1 = 0.0, d2 = 0.0, d3 = 0.0;
#pragma unroll
        for (int l = 0; l < NGL; ++l) {
            const int p = rb + l;
            const double dl = sD[xi * NGL + l];
            double f1, f2, f3;
            pair_flux_raw<false>(g, h, hu, hv, uL, vL, h2L, ye, xe, sh[p], shu[p], shv[p], su[p], sv[p], sh2[p], sYe[p],
                                 sXe[p], f1, f2, f3);
            d1 += dl * f1; d2 += dl * f2; d3 += dl * f3;
        }
#pragma unroll
        for (int l = 0; l < NGL; ++l) {
            const int p = cb + l * NGL;
            const double dl = sD[eta * NGL + l];
            double g1, g2, g3;
            pair_flux_raw<true>(g, h, hu, hv, uL, vL, h2L, yx, xx, sh[p], shu[p], shv[p], su[p], sv[p], sh2[p], sYx[p],
                                sXx[p], g1, g2, g3);
            d1 += dl * g1; d2 += dl * g2; d3 += dl * g3;
        }
        d1 *= 0.25;
        d2 *= 0.125;
        d3 *= 0.125;
        double r0 = -J * d1;
        double r1 = -J * d2 - a.c.g * h * bx;
        double r2 = -J * d3 - a.c.g * h * by;
        if (GEN == 1 && a.dry && a.dry[e])
            pd_volume<NGL>(a.c, a.Dc, a.Dup, a.Ddn, sh + el * N2, a.Bn + (long)e * N2, eta, xi, ye, yx, xe, xx, J, r1,
                           r2);
        // lift: sides 0/2 first, then 1/3 (-ms * flux; DBSurf1/2 are zero)
        const double db = 0.0;
#pragma unroll
        for (int pass = 0; pass < 2; ++pass) {
            if (has[pass]) {
                r0 += f[pass][0] * J;
                r1 += J * f[pass][1] + J * db;
                r2 += J * f[pass][2] + J * db;
            }
        }
        if (GEN == 1 && a.conv) add_conv_source(a, a.st[ins], xid, bx, by, r0, r1, r2);
        if (a.mode == 2 || to_list) {
            a.Qt[qid] = r0; a.Qt[qid + N2] = r1; a.Qt[qid + 2 * N2] = r2;
        } else {
            double q0, q1, q2;
            if (a.mode == 0) {
                const double g0 = a.rkA * o0 + r0;
                const double g1 = a.rkA * o1 + r1;
                const double g2 = a.rkA * o2 + r2;
                a.gRK[qid] = g0; a.gRK[qid + N2] = g1; a.gRK[qid + 2 * N2] = g2;
                q0 = h + a.rkC * dt * g0;
                q1 = hu + a.rkC * dt * g1;
                q2 = hv + a.rkC * dt * g2;
            } else {
                q0 = a.rkA * o0 + a.rkB * h + a.rkC * dt * r0;
                q1 = a.rkA * o1 + a.rkB * hu + a.rkC * dt * r1;
                q2 = a.rkA * o2 + a.rkB * hv + a.rkC * dt * r2;
            }
            a.q[qid] = q0; a.q[qid + N2] = q1; a.q[qid + 2 * N2] = q2;
            if (a.lam) lam = node_lambda(a.c, q0, q1, q2);
        }
    }
    if (a.lam) warp_lambda<ElemShape<NGL>::THREADS>(lam, active && !to_list, ins, a.st);
}

}  // namespace esdg
