// Adjoint of ElmGMR's residual: lambda^T d res / d(y_alpha, ac_alpha, mu,
// coef1, coef2), exact (no counterpart in the reference, which has no
// adjoint).
//
// res is the vector ElmGMR assembles (flowsolver/src/elmgmr.f90:82-555):
// the interior SUPG/PSPG residual (e3ivar/e3stab/e3Res, e3ivar.f90:99-198,
// e3stab.f90:83-133, e3res.f90:94-286) with the viscous-flux projection
// qres (AsIq/qpbc, asiq.f90:52-70, qpbc.f90:67-71), the boundary residual
// (e3b/e3bvar, e3b.f90:112-470), the outlet coupling p_k NABI with
// p_k = -(Q_k coef1_k) - coef2_k (elmgmr.f90:1271-1330) and bc3Res.
//
// The element tangent ElmGMR assembles (e3LHS) is the reference's
// approximate Jacobian: it omits the derivatives of tauM, tauC, tauBar and
// of uBar and the viscous-flux projection.  The adjoint needs the exact
// transposed Jacobian, so each tet's contraction J = sum_a lambda_a . rl_a is
// differentiated by hand in reverse: per quadrature point the forward
// quantities once, then their cotangents, about twice the residual's
// arithmetic for all 32 local inputs together -- y_alpha (4 nodes x p,u,v,w),
// ac_alpha (4 x 3), div q (3: on a linear tet div q = sum_n dN_n . q_n is an
// element constant) and mu.  The cotangent of div q goes to the nodal qres
// through dN, and from qres through the transposed lumped projection back to
// u and mu.
//
// Scatter as in the assembly: the element kernels write records (the work
// space of ElmGMR's records), node passes sum them per node in a fixed order;
// mu's cotangent is summed per block and over the blocks in order.  Only the
// boundary faces and outlet nodes, few, are added with atomics.
//
// Bound by the record traffic (416 B written per tet, 192 B read per tet and
// node) and the latency of the element kernel's gathers.  On the 1M-tet
// 3-outlet cylinder the whole product took 8.3 ms with forward-mode dual
// numbers (four passes of eight directions, 2.2 KB of stack per thread, 64
// FP64 atomics per tet).
#include <vector>

#include "common.cuh"

namespace crimson {

int elmgmr_device(crimson_ctx* c, const double* d_y, const double* d_ac, const double* coef1, const double* coef2,
                  double* d_res, double* d_lhsK, double* d_lhsP, int lhs, float* d_lhs32 = nullptr);

// ---------------------------------------------------------------------------
// Element tables and settings
// ---------------------------------------------------------------------------
struct AdjConst {
    double shp[4][4];   // shp[q][n] at the 4-point rule (symtet.c, uniformP.c:22-40)
    double Qwt;         // (1/4) * (4/3) (genint.f90:85)
    double SN[4];       // sum_q shp[q][n]
    double shpb[3][4];  // boundary 3-point rule
    double Qwtb;
};

struct AdjParams {
    double rho, Dtgl, dtsfct, taucfct, stabflux;
    int idiff;
};

static AdjConst make_adj_consts() {
    const double A4 = 0.5854101966249685, B4 = 0.1381966011250150;
    const double rstw4[4][3] = {{A4, B4, B4}, {B4, A4, B4}, {B4, B4, A4}, {B4, B4, B4}};
    AdjConst k{};
    for (int q = 0; q < 4; ++q) {
        k.shp[q][0] = rstw4[q][0];
        k.shp[q][1] = rstw4[q][1];
        k.shp[q][2] = rstw4[q][2];
        k.shp[q][3] = 1.0e0 - rstw4[q][0] - rstw4[q][1] - rstw4[q][2];
    }
    k.Qwt = (4.0 / 3.0) * 0.25;
    for (int a = 0; a < 4; ++a) {
        k.SN[a] = 0.0;
        for (int q = 0; q < 4; ++q) k.SN[a] += k.shp[q][a];
    }
    const double B3 = 0.666666666666667, C3 = 0.166666666666667, A3 = 0.3333333333333330000000000000000000;
    const double rst3[3][3] = {{B3, C3, C3}, {C3, B3, C3}, {C3, C3, B3}};
    for (int q = 0; q < 3; ++q) {
        k.shpb[q][0] = rst3[q][0];
        k.shpb[q][1] = rst3[q][1];
        k.shpb[q][2] = rst3[q][2];
        k.shpb[q][3] = 1.0e0 - rst3[q][0] - rst3[q][1] - rst3[q][2];
    }
    k.Qwtb = 2.0 * A3;
    return k;
}

// e3metric for a linear tet (e3metric.f90:26-81): dxidx, shg = dN/dx, WdetJ
__device__ __forceinline__ void adj_metric(const double xl[4][3], double Qwt, double dxidx[3][3], double shg[4][3],
                                           double* WdetJ) {
    double d[3][3];
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) d[i][j] = 0.5 * xl[j][i] - 0.5 * xl[3][i];
    dxidx[0][0] = d[1][1] * d[2][2] - d[2][1] * d[1][2];
    dxidx[0][1] = d[2][1] * d[0][2] - d[0][1] * d[2][2];
    dxidx[0][2] = d[0][1] * d[1][2] - d[0][2] * d[1][1];
    const double tmp = 1.0 / (dxidx[0][0] * d[0][0] + dxidx[0][1] * d[1][0] + dxidx[0][2] * d[2][0]);
    dxidx[0][0] *= tmp;
    dxidx[0][1] *= tmp;
    dxidx[0][2] *= tmp;
    dxidx[1][0] = (d[1][2] * d[2][0] - d[1][0] * d[2][2]) * tmp;
    dxidx[1][1] = (d[0][0] * d[2][2] - d[2][0] * d[0][2]) * tmp;
    dxidx[1][2] = (d[1][0] * d[0][2] - d[0][0] * d[1][2]) * tmp;
    dxidx[2][0] = (d[1][0] * d[2][1] - d[1][1] * d[2][0]) * tmp;
    dxidx[2][1] = (d[2][0] * d[0][1] - d[0][0] * d[2][1]) * tmp;
    dxidx[2][2] = (d[0][0] * d[1][1] - d[0][1] * d[1][0]) * tmp;
    *WdetJ = Qwt / tmp;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        shg[0][k] = 0.5 * dxidx[0][k];
        shg[1][k] = 0.5 * dxidx[1][k];
        shg[2][k] = 0.5 * dxidx[2][k];
        shg[3][k] = -0.5 * dxidx[0][k] - 0.5 * dxidx[1][k] - 0.5 * dxidx[2][k];
    }
}

// e3gijd, tet branch (e3stab.f90:487-528)
__device__ __forceinline__ void adj_gijd(const double dx[3][3], double g[6]) {
    const double c1 = 1.259921049894873e+00;
    const double c2 = 6.299605249474365e-01;
    double t1, t2, t3;
    t1 = c1 * dx[0][0] + c2 * (dx[1][0] + dx[2][0]);
    t2 = c1 * dx[1][0] + c2 * (dx[0][0] + dx[2][0]);
    t3 = c1 * dx[2][0] + c2 * (dx[0][0] + dx[1][0]);
    g[0] = dx[0][0] * t1 + dx[1][0] * t2 + dx[2][0] * t3;
    t1 = c1 * dx[0][1] + c2 * (dx[1][1] + dx[2][1]);
    t2 = c1 * dx[1][1] + c2 * (dx[0][1] + dx[2][1]);
    t3 = c1 * dx[2][1] + c2 * (dx[0][1] + dx[1][1]);
    g[1] = dx[0][1] * t1 + dx[1][1] * t2 + dx[2][1] * t3;
    g[3] = dx[0][0] * t1 + dx[1][0] * t2 + dx[2][0] * t3;
    t1 = c1 * dx[0][2] + c2 * (dx[1][2] + dx[2][2]);
    t2 = c1 * dx[1][2] + c2 * (dx[0][2] + dx[2][2]);
    t3 = c1 * dx[2][2] + c2 * (dx[0][2] + dx[1][2]);
    g[2] = dx[0][2] * t1 + dx[1][2] * t2 + dx[2][2] * t3;
    g[4] = dx[0][1] * t1 + dx[1][1] * t2 + dx[2][1] * t3;
    g[5] = dx[0][0] * t1 + dx[1][0] * t2 + dx[2][0] * t3;
}

// ---------------------------------------------------------------------------
// Kernels
// ---------------------------------------------------------------------------
// Element record (the first doubles of ElmGMR's): at 8 a the cotangents of
// node a's (u, v, w, p) and (ax, ay, az, 0); grad N_a at 32 + 4 a; that of
// div q at 48.
constexpr int kAdjRS = 52;
constexpr int kAdjBlocksPerSM = 8;   // cap of the element kernels' grids (partial sums of mu's cotangent)

// lambda with the rows bc3Res zeroes set to zero (node-major (4, n))
__global__ void k_adj_mask(const int* __restrict__ iBC, const double* __restrict__ lam, double* __restrict__ out,
                           int n) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int b = iBC[i];
        const double* l = lam + 4 * (size_t)i;
        double* o = out + 4 * (size_t)i;
        const bool vel = ((b >> 3) & 7) == 7 || ((b >> 11) & 1);
        o[0] = vel ? 0.0 : l[0];
        o[1] = vel ? 0.0 : l[1];
        o[2] = vel ? 0.0 : l[2];
        o[3] = ((b >> 2) & 1) ? 0.0 : l[3];
    }
}

// Metric tensor product G v, G from gijd = (11, 22, 33, 12, 23, 13).
__device__ __forceinline__ void adj_gv(const double G[6], const double v[3], double o[3]) {
    o[0] = G[0] * v[0] + G[3] * v[1] + G[5] * v[2];
    o[1] = G[3] * v[0] + G[1] * v[1] + G[4] * v[2];
    o[2] = G[5] * v[0] + G[4] * v[1] + G[2] * v[2];
}

// Sum over an element's four lanes (fixed butterfly).
__device__ __forceinline__ double adj_quad_sum(double v) {
    v += __shfl_xor_sync(0xffffffffu, v, 1);
    v += __shfl_xor_sync(0xffffffffu, v, 2);
    return v;
}

// Interior cotangents, four lanes per tet: lane q evaluates quadrature point
// q, lane a writes node a (one lane per tet holds the sums of all points and
// nodes in 255 registers and spills).  Forward per point: u, ac, p,
//   L_i = rho (ac_i + u . grad u_i) + p,i - divq_i,   F = sqrt(. + u.Gu + .)
//   tauM = 1/F, tauC = kC F, B = L.GL, tauB = tauM / sqrt(B)
//   uB = u - tauM L / rho, h_i = L . grad u_i, rN_i = rho (ac_i + uB . grad u_i)
//   rG_ij = mu (u_i,j + u_j,i) + tauM L_i u_j + tauB h_i L_j + d_ij (tauC div u - p)
//   J = W sum_q [ Lc . uB - l . rN - Lm_ij rG_ij ]
// with Lc_j = sum_a lambda_a4 N_a,j, Lm_ij = sum_a lambda_ai N_a,j (element
// constants) and l_i = sum_a lambda_ai N_a.
__global__ void __launch_bounds__(128) k_adj_interior(const int4* __restrict__ ien, const double4* __restrict__ x,
                                                      const double4* __restrict__ y, const double4* __restrict__ ac,
                                                      const double* __restrict__ qres, const double4* __restrict__ lam,
                                                      int nelem, AdjConst C, AdjParams P, double mu,
                                                      double* __restrict__ erec, double* __restrict__ mupart) {
    __shared__ double sm[32];
    const int q = threadIdx.x & 3;
    double mub = 0.0;
    const double rho = P.rho, rinv = 1.0 / rho, dts = P.Dtgl * P.dtsfct;
    double N[4];
#pragma unroll
    for (int a = 0; a < 4; ++a) N[a] = C.shp[q][a];
    // block-uniform loop: the shuffles always see all lanes; lanes past the
    // last tet work on the last one and write nothing
    for (int e0 = blockIdx.x * (blockDim.x >> 2); e0 < nelem; e0 += gridDim.x * (blockDim.x >> 2)) {
        const bool live = e0 + (int)(threadIdx.x >> 2) < nelem;
        const int e = live ? e0 + (int)(threadIdx.x >> 2) : nelem - 1;
        const int4 nn = ien[e];
        const int nd[4] = {nn.x, nn.y, nn.z, nn.w};
        double shg[4][3], W, G[6];
        {
            double xl[4][3], dxidx[3][3];
#pragma unroll
            for (int a = 0; a < 4; ++a) {
                const double4 xx = ld32(x + nd[a]);
                xl[a][0] = xx.x;
                xl[a][1] = xx.y;
                xl[a][2] = xx.z;
            }
            adj_metric(xl, C.Qwt, dxidx, shg, &W);
            adj_gijd(dxidx, G);
        }
        double Lm[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}}, Lc[3] = {0, 0, 0};
        double g[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}};   // g[k][i] = u_i,k
        double u[3] = {0, 0, 0}, L[3] = {0, 0, 0}, l[3] = {0, 0, 0}, res[3] = {0, 0, 0};
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            const double4 ll = ld32(lam + nd[a]), yy = y[nd[a]], aa = ac[nd[a]];
            const double l3[3] = {ll.x, ll.y, ll.z}, u3[3] = {yy.x, yy.y, yy.z}, a3[3] = {aa.x, aa.y, aa.z};
#pragma unroll
            for (int j = 0; j < 3; ++j) {
                u[j] += N[a] * u3[j];
                L[j] += N[a] * a3[j];   // ac at the point, for now
                l[j] += N[a] * l3[j];
                Lc[j] += ll.w * shg[a][j];
                res[j] += shg[a][j] * yy.w;   // grad p - div q
#pragma unroll
                for (int i = 0; i < 3; ++i) {
                    Lm[i][j] += l3[i] * shg[a][j];
                    g[j][i] += shg[a][j] * u3[i];
                }
            }
        }
        if (P.idiff >= 1) {
            // lane a gathers node a's projected flux
            const double* f = qres + 9 * (size_t)(q == 0 ? nd[0] : (q == 1 ? nd[1] : (q == 2 ? nd[2] : nd[3])));
            const double s0 = q == 0 ? shg[0][0] : (q == 1 ? shg[1][0] : (q == 2 ? shg[2][0] : shg[3][0]));
            const double s1 = q == 0 ? shg[0][1] : (q == 1 ? shg[1][1] : (q == 2 ? shg[2][1] : shg[3][1]));
            const double s2 = q == 0 ? shg[0][2] : (q == 1 ? shg[1][2] : (q == 2 ? shg[2][2] : shg[3][2]));
#pragma unroll
            for (int i = 0; i < 3; ++i) res[i] -= adj_quad_sum(s0 * f[i] + s1 * f[i + 3] + s2 * f[i + 6]);
        }
        const double gg = G[0] * G[0] + G[1] * G[1] + G[2] * G[2] + 2.0 * (G[3] * G[3] + G[4] * G[4] + G[5] * G[5]);
        const double kC = rho * 0.125 / (G[0] + G[1] + G[2]) * (P.taucfct / P.dtsfct);
        const double f0 = (2.0 * dts) * (2.0 * dts) + 36.0 * (mu * rinv) * (mu * rinv) * gg;
        const double divu = g[0][0] + g[1][1] + g[2][2], trL = Lm[0][0] + Lm[1][1] + Lm[2][2];
#pragma unroll
        for (int i = 0; i < 3; ++i) L[i] = (L[i] + u[0] * g[0][i] + u[1] * g[1][i] + u[2] * g[2][i]) * rho + res[i];
        double Gu[3], GL[3];
        adj_gv(G, u, Gu);
        adj_gv(G, L, GL);
        const double F = sqrt(f0 + u[0] * Gu[0] + u[1] * Gu[1] + u[2] * Gu[2]);
        const double tauM = 1.0 / F, tauC = kC * F;
        const double B = L[0] * GL[0] + L[1] * GL[1] + L[2] * GL[2];
        const double rB = B != 0.0 ? 1.0 / sqrt(B) : 0.0;
        const double tauB = tauM * rB;
        double h[3], ml[3];   // ml_i: minus the cotangent of tauB h_i
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            h[i] = L[0] * g[0][i] + L[1] * g[1][i] + L[2] * g[2][i];
            ml[i] = Lm[i][0] * L[0] + Lm[i][1] * L[1] + Lm[i][2] * L[2];
        }
        // cotangents (without W) of u, L, ac, the gradients gb[k][i], tau and mu at this point
        double ub[3], Lb[3], acb[3], gb[3][3], tauMb = 0.0, tauBb = 0.0, mb = 0.0;
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            const double mu_i = Lm[i][0] * u[0] + Lm[i][1] * u[1] + Lm[i][2] * u[2];
            const double lt = Lm[0][i] * L[0] + Lm[1][i] * L[1] + Lm[2][i] * L[2];
            const double ht = Lm[0][i] * h[0] + Lm[1][i] * h[1] + Lm[2][i] * h[2];
            const double uBb = Lc[i] - rho * (l[0] * g[i][0] + l[1] * g[i][1] + l[2] * g[i][2]);
            ub[i] = uBb - tauM * lt;
            Lb[i] = -tauM * mu_i - tauB * (ht + g[i][0] * ml[0] + g[i][1] * ml[1] + g[i][2] * ml[2]) - tauM * rinv * uBb;
            tauMb -= L[i] * mu_i + uBb * L[i] * rinv;
            tauBb -= ml[i] * h[i];
            acb[i] = -rho * l[i];
        }
        tauMb += tauBb * rB;
        const double Bb = -0.5 * tauBb * tauB * rB * rB;
        // F: tauM = 1/F, tauC = kC F (cotangent -trL div u); F = sqrt(s)
        const double sb = 0.5 * tauM * (-tauMb * tauM * tauM - kC * trL * divu);
        mb = sb * 72.0 * mu * rinv * rinv * gg;
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            Lb[i] += 2.0 * Bb * GL[i];
            ub[i] += 2.0 * sb * Gu[i];
            acb[i] += rho * Lb[i];
        }
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const double uBk = u[k] - tauM * L[k] * rinv;
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                mb -= Lm[i][k] * (g[k][i] + g[i][k]);
                gb[k][i] = -mu * (Lm[i][k] + Lm[k][i]) - L[k] * tauB * ml[i] - rho * l[i] * uBk + rho * u[k] * Lb[i];
                ub[k] += rho * Lb[i] * g[k][i];
            }
            gb[k][k] -= trL * tauC;
        }
        // over the points: gradients' cotangents, div q's (-Lb), mu's
#pragma unroll
        for (int k = 0; k < 3; ++k)
#pragma unroll
            for (int i = 0; i < 3; ++i) gb[k][i] = adj_quad_sum(gb[k][i]);
        double gpb[3];
#pragma unroll
        for (int i = 0; i < 3; ++i) gpb[i] = adj_quad_sum(Lb[i]);
        // node a = q: sum over the points p of N_a(p) times the points' cotangents
        double yb[3] = {0, 0, 0}, ab[3] = {0, 0, 0};
#pragma unroll
        for (int p = 0; p < 4; ++p) {
            const double Na = C.shp[p][q];
            const int src = (threadIdx.x & 28) | p;
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                yb[i] += Na * __shfl_sync(0xffffffffu, ub[i], src);
                ab[i] += Na * __shfl_sync(0xffffffffu, acb[i], src);
            }
        }
        if (!live) continue;
        const double s[3] = {q == 0 ? shg[0][0] : (q == 1 ? shg[1][0] : (q == 2 ? shg[2][0] : shg[3][0])),
                             q == 0 ? shg[0][1] : (q == 1 ? shg[1][1] : (q == 2 ? shg[2][1] : shg[3][1])),
                             q == 0 ? shg[0][2] : (q == 1 ? shg[1][2] : (q == 2 ? shg[2][2] : shg[3][2]))};
        double4* r4 = reinterpret_cast<double4*>(erec + (size_t)kAdjRS * e);
        double o[3];
#pragma unroll
        for (int i = 0; i < 3; ++i) o[i] = W * (yb[i] + s[0] * gb[0][i] + s[1] * gb[1][i] + s[2] * gb[2][i]);
        st32(r4 + 2 * q, make_double4(o[0], o[1], o[2],
                                      W * (C.SN[q] * trL + s[0] * gpb[0] + s[1] * gpb[1] + s[2] * gpb[2])));
        st32(r4 + 2 * q + 1, make_double4(W * ab[0], W * ab[1], W * ab[2], 0.0));
        st32(r4 + 8 + q, make_double4(s[0], s[1], s[2], 0.0));
        if (q == 0) st32(r4 + 12, make_double4(-W * gpb[0], -W * gpb[1], -W * gpb[2], 0.0));
        mub += W * mb;
    }
    mub = block_sum(mub, sm);
    if (threadIdx.x == 0) mupart[blockIdx.x] = mub;
}

// Lanes per node in the node passes, combined in a fixed butterfly.
constexpr int kAdjLanes = 4;
__device__ __forceinline__ double adj_lanes_sum(double v) {
#pragma unroll
    for (int o = kAdjLanes / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Cotangent of qres over the elements at each node, times 1 / rmass (qpbc):
// div q_i = sum_a sum_j N_a,j q_a(i + 3 j).
__global__ void __launch_bounds__(256) k_adj_qnode(const int* __restrict__ diag, const int* __restrict__ soff,
                                                   const int* __restrict__ slist, const double* __restrict__ erec,
                                                   const double* __restrict__ rmass, int nshg,
                                                   double* __restrict__ qbar) {
    constexpr int NPW = 32 / kAdjLanes;
    const int lane = threadIdx.x & 31, sub = lane % kAdjLanes;
    const long long warp = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const long long nwarp = ((long long)gridDim.x * blockDim.x) >> 5;
    for (long long i0 = warp * NPW; i0 < nshg; i0 += nwarp * NPW) {
        const long long ig = i0 + lane / kAdjLanes;
        const bool valid = ig < nshg;
        const int i = valid ? (int)ig : nshg - 1;
        const int d = diag[i], p1 = soff[d + 1];
        double q[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
        for (int p = soff[d] + sub; p < p1; p += kAdjLanes) {
            const int t = slist[p];
            const double4* r4 = reinterpret_cast<const double4*>(erec + (size_t)kAdjRS * (t >> 4));
            const double4 s = ld32(r4 + 8 + ((t >> 2) & 3)), v = ld32(r4 + 12);
            q[0] += s.x * v.x;
            q[1] += s.x * v.y;
            q[2] += s.x * v.z;
            q[3] += s.y * v.x;
            q[4] += s.y * v.y;
            q[5] += s.y * v.z;
            q[6] += s.z * v.x;
            q[7] += s.z * v.y;
            q[8] += s.z * v.z;
        }
#pragma unroll
        for (int k = 0; k < 9; ++k) q[k] = adj_lanes_sum(q[k]);
        if (!valid || sub != 0) continue;
        const double r = rmass[i];
#pragma unroll
        for (int k = 0; k < 9; ++k) qbar[9 * (size_t)i + k] = r * q[k];
    }
}

// Transposed lumped projection (AsIq + qpbc): qres_a = (sum_e W SN_a qdi_e) /
// rmass_a with qdi = mu (grad u + grad u^T).  Per tet the cotangent of grad u
// (symmetric: 11, 22, 33, 12, 13, 23 of an 8-double record) and of mu.
__global__ void __launch_bounds__(128) k_adj_asiq(const int4* __restrict__ ien, const double4* __restrict__ x,
                                                  const double4* __restrict__ y, const double* __restrict__ qbar,
                                                  int nelem, AdjConst C, double mu, double* __restrict__ grec,
                                                  double* __restrict__ mupart) {
    __shared__ double sm[32];
    double mub = 0.0;
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < nelem; e += gridDim.x * blockDim.x) {
        const int4 nn = ien[e];
        const int nd[4] = {nn.x, nn.y, nn.z, nn.w};
        double xl[4][3], ul[4][3];
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            const double4 xx = ld32(x + nd[a]);
            const double4 yy = y[nd[a]];
            xl[a][0] = xx.x;
            xl[a][1] = xx.y;
            xl[a][2] = xx.z;
            ul[a][0] = yy.x;
            ul[a][1] = yy.y;
            ul[a][2] = yy.z;
        }
        double dxidx[3][3], shg[4][3], W;
        adj_metric(xl, C.Qwt, dxidx, shg, &W);
        double qb[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            const double w = W * C.SN[a];
            const double* q = qbar + 9 * (size_t)nd[a];
#pragma unroll
            for (int k = 0; k < 9; ++k) qb[k] += w * q[k];
        }
        double g[3][3];  // g[k][i] = d u_i / d x_k
#pragma unroll
        for (int k = 0; k < 3; ++k)
#pragma unroll
            for (int i = 0; i < 3; ++i)
                g[k][i] = shg[0][k] * ul[0][i] + shg[1][k] * ul[1][i] + shg[2][k] * ul[2][i] + shg[3][k] * ul[3][i];
        const double s12 = qb[1] + qb[3], s13 = qb[2] + qb[6], s23 = qb[5] + qb[7];
        mub += 2.0 * (qb[0] * g[0][0] + qb[4] * g[1][1] + qb[8] * g[2][2]) + s12 * (g[0][1] + g[1][0]) +
               s13 * (g[0][2] + g[2][0]) + s23 * (g[1][2] + g[2][1]);
        double4* r = reinterpret_cast<double4*>(grec + 8 * (size_t)e);
        st32(r, make_double4(2.0 * mu * qb[0], 2.0 * mu * qb[4], 2.0 * mu * qb[8], mu * s12));
        st32(r + 1, make_double4(mu * s13, mu * s23, 0.0, 0.0));
    }
    mub = block_sum(mub, sm);
    if (threadIdx.x == 0) mupart[blockIdx.x] = mub;
}

// ybar and abar of every node from its elements' records (and the projection
// records grec, when there are).
__global__ void __launch_bounds__(256) k_adj_node(const int* __restrict__ diag, const int* __restrict__ soff,
                                                  const int* __restrict__ slist, const double* __restrict__ erec,
                                                  const double* __restrict__ grec, int nshg, double* __restrict__ ybar,
                                                  double* __restrict__ abar) {
    static_assert(kAdjLanes == 4, "a node's lanes write its four components");
    constexpr int NPW = 32 / kAdjLanes;
    const int lane = threadIdx.x & 31, sub = lane % kAdjLanes;
    const long long warp = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const long long nwarp = ((long long)gridDim.x * blockDim.x) >> 5;
    for (long long i0 = warp * NPW; i0 < nshg; i0 += nwarp * NPW) {
        const long long ig = i0 + lane / kAdjLanes;
        const bool valid = ig < nshg;
        const int i = valid ? (int)ig : nshg - 1;
        const int d = diag[i], p1 = soff[d + 1];
        double v[7] = {0, 0, 0, 0, 0, 0, 0};
        for (int p = soff[d] + sub; p < p1; p += kAdjLanes) {
            const int t = slist[p], a = (t >> 2) & 3;
            const double4* r4 = reinterpret_cast<const double4*>(erec + (size_t)kAdjRS * (t >> 4));
            const double4 yy = ld32(r4 + 2 * a), aa = ld32(r4 + 2 * a + 1);
            v[0] += yy.x;
            v[1] += yy.y;
            v[2] += yy.z;
            v[3] += yy.w;
            v[4] += aa.x;
            v[5] += aa.y;
            v[6] += aa.z;
            if (grec) {
                const double4* q4 = reinterpret_cast<const double4*>(grec + 8 * (size_t)(t >> 4));
                const double4 s = ld32(r4 + 8 + a), A = ld32(q4), B = ld32(q4 + 1);
                v[0] += s.x * A.x + s.y * A.w + s.z * B.x;
                v[1] += s.x * A.w + s.y * A.y + s.z * B.y;
                v[2] += s.x * B.x + s.y * B.y + s.z * A.z;
            }
        }
#pragma unroll
        for (int k = 0; k < 7; ++k) v[k] = adj_lanes_sum(v[k]);
        if (!valid) continue;
        // lane sub writes component sub: the caller's arrays, 8-byte aligned
        ybar[4 * (size_t)i + sub] = sub == 0 ? v[0] : (sub == 1 ? v[1] : (sub == 2 ? v[2] : v[3]));
        abar[4 * (size_t)i + sub] = sub == 0 ? v[4] : (sub == 1 ? v[5] : (sub == 2 ? v[6] : 0.0));
    }
}

// Boundary-face cotangents (e3b/e3bvar rigid wall as k_asbmfg forms it),
// nodes 0..2 on the face, node 3 interior; added to ybar after the node pass.
__global__ void __launch_bounds__(128) k_adj_faces(const int4* __restrict__ ienb, const int* __restrict__ iBCB,
                                                   const double4* __restrict__ x, const double4* __restrict__ y,
                                                   const double4* __restrict__ lam, int nface, AdjConst C, AdjParams P,
                                                   double mu, double* __restrict__ ybar,
                                                   double* __restrict__ mupart) {
    __shared__ double sm[32];
    double mub = 0.0;
    for (int f = blockIdx.x * blockDim.x + threadIdx.x; f < nface; f += gridDim.x * blockDim.x) {
        const int4 nn = ienb[f];
        const int nd[4] = {nn.x, nn.y, nn.z, nn.w};
        double xl[4][3], yl[4][4], lm[3][4];
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            const double4 xx = x[nd[a]];
            const double4 yy = y[nd[a]];
            xl[a][0] = xx.x;
            xl[a][1] = xx.y;
            xl[a][2] = xx.z;
            yl[a][0] = yy.x;
            yl[a][1] = yy.y;
            yl[a][2] = yy.z;
            yl[a][3] = yy.w;
        }
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const double4 ll = lam[nd[a]];
            lm[a][0] = ll.x;
            lm[a][1] = ll.y;
            lm[a][2] = ll.z;
            lm[a][3] = ll.w;
        }
        const int bits = iBCB[f];
        double dxidx[3][3], shg[4][3], Wtmp;
        adj_metric(xl, C.Qwt, dxidx, shg, &Wtmp);
        double v1[3], v2[3];
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            v1[i] = xl[1][i] - xl[0][i];
            v2[i] = xl[2][i] - xl[0][i];
        }
        const double t1 = v1[1] * v2[2] - v2[1] * v1[2];
        const double t2 = v2[0] * v1[2] - v1[0] * v2[2];
        const double t3 = v1[0] * v2[1] - v2[0] * v1[1];
        const double temp = 1.0 / sqrt(t1 * t1 + t2 * t2 + t3 * t3);
        const double bn[3] = {t1 * temp, t2 * temp, t3 * temp};
        const double Wb = C.Qwtb / (4.0 * temp);
        // natural pressure (bit 1) replaces the pressure, bit 2 the traction,
        // bit 4 both, bit 0 the normal velocity of the continuity row
        const bool pres_live = !(bits & 2) && !(bits & 16), tt_live = !(bits & 4) && !(bits & 16);
        double taub[3] = {0, 0, 0}, ybn[3][4] = {{0, 0, 0, 0}, {0, 0, 0, 0}, {0, 0, 0, 0}};
        for (int q = 0; q < 3; ++q) {
            const double* Nb = C.shpb[q];
            double u[3], l[4], pres = 0.0;
#pragma unroll
            for (int i = 0; i < 3; ++i) u[i] = Nb[0] * yl[0][i] + Nb[1] * yl[1][i] + Nb[2] * yl[2][i];
#pragma unroll
            for (int d = 0; d < 4; ++d) l[d] = Nb[0] * lm[0][d] + Nb[1] * lm[1][d] + Nb[2] * lm[2][d];
            const double unm = bn[0] * u[0] + bn[1] * u[1] + bn[2] * u[2];
            const bool back = (bits & 2) && unm < 0.0;
            const double sf = P.stabflux * P.rho * (back ? unm : 0.0);
            // rNa_i = (bn_i pres - tt_i - stabflux rho unm_copy u_i) Wb, rNa_4 = unm Wb; J = -l . rNa
            double rb[3], presb = 0.0, tnb = 0.0, unb = bits & 1 ? 0.0 : -l[3] * Wb;
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                rb[i] = -l[i] * Wb;
                presb += bn[i] * rb[i];
                if (back) unb -= P.stabflux * P.rho * u[i] * rb[i];
            }
            if (!pres_live) presb = 0.0;
            tnb -= presb;
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                const double ttb = tt_live ? -rb[i] : 0.0;
                taub[i] += ttb;
                tnb -= bn[i] * ttb;
            }
            pres = presb;
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                taub[i] += bn[i] * tnb;
                const double ub = bn[i] * unb - sf * rb[i];
#pragma unroll
                for (int n = 0; n < 3; ++n) ybn[n][i] += Nb[n] * ub;
            }
#pragma unroll
            for (int n = 0; n < 3; ++n) ybn[n][3] += Nb[n] * pres;
        }
        // tau_i = mu sum_k bn_k (u_i,k + u_k,i)
        double gb[3][3];
#pragma unroll
        for (int k = 0; k < 3; ++k)
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                gb[k][i] = mu * (bn[k] * taub[i] + bn[i] * taub[k]);
                const double g = shg[0][k] * yl[0][i] + shg[1][k] * yl[1][i] + shg[2][k] * yl[2][i] + shg[3][k] * yl[3][i];
                mub += (bn[k] * taub[i] + bn[i] * taub[k]) * g;
            }
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            double* o = ybar + 4 * (size_t)nd[a];
#pragma unroll
            for (int i = 0; i < 3; ++i)
                atomicAdd(o + i, (a < 3 ? ybn[a < 3 ? a : 0][i] : 0.0) + shg[a][0] * gb[0][i] + shg[a][1] * gb[1][i] +
                                     shg[a][2] * gb[2][i]);
            if (a < 3) atomicAdd(o + 3, ybn[a < 3 ? a : 0][3]);
        }
    }
    mub = block_sum(mub, sm);
    if (threadIdx.x == 0) mupart[blockIdx.x] = mub;
}

// out = sum of the n partial sums, in order
__global__ void k_adj_sum(const double* __restrict__ part, int n, double* __restrict__ out) {
    __shared__ double sm[32];
    double s = 0.0;
    for (int t = threadIdx.x; t < n; t += blockDim.x) s += part[t];
    s = block_sum(s, sm);
    if (threadIdx.x == 0) *out = s;
}

// s_k = sum over outlet k's nodes of NABI . v (v = y or lambda), fixed order
__global__ void k_adj_flow(const int* __restrict__ onodes, const int* __restrict__ off,
                           const double4* __restrict__ onabi, const double4* __restrict__ v, double* __restrict__ s) {
    __shared__ double sm[32];
    const int k = blockIdx.x;
    double t = 0.0;
    for (int j = off[k] + threadIdx.x; j < off[k + 1]; j += blockDim.x) {
        const double4 nb = onabi[j];
        const double4 vv = v[onodes[j]];
        t += nb.x * vv.x + nb.y * vv.y + nb.z * vv.z;
    }
    t = block_sum(t, sm);
    if (threadIdx.x == 0) s[k] = t;
}

// ybar(vel) -= coef1_k s_k NABI over outlet k's nodes (d p_k / d u)
__global__ void k_adj_pvsq(const int* __restrict__ onodes, const int* __restrict__ off,
                           const double4* __restrict__ onabi, const double* __restrict__ s,
                           const double* __restrict__ coef1, int ncoupled, double* __restrict__ ybar) {
    const int k = blockIdx.y;
    const double f = -coef1[k] * s[k];
    for (int j = off[k] + blockIdx.x * blockDim.x + threadIdx.x; j < off[k + 1]; j += gridDim.x * blockDim.x) {
        const double4 nb = onabi[j];
        double* r = ybar + 4 * (size_t)onodes[j];
        atomicAdd(r + 0, f * nb.x);
        atomicAdd(r + 1, f * nb.y);
        atomicAdd(r + 2, f * nb.z);
    }
}

int elmgmr_vjp(crimson_ctx* c, const double* d_y, const double* d_ac, const double* coef1, const double* coef2,
               const double* d_lam, double* d_res, double* d_ybar, double* d_abar, double* mubar, double* c1bar,
               double* c2bar) {
    cudaStream_t s = c->stream;
    const int n = c->nshg;
    const crimson_params& p = c->p;
    // primal residual at (y, ac): also leaves qres and 1/rmass in the context
    CR_CHECK(c->adj_res.alloc(4 * (size_t)n));
    CR_CHECK(elmgmr_device(c, d_y, d_ac, coef1, coef2, d_res ? d_res : c->adj_res.p, nullptr, nullptr, 0));
    const int nc = c->ncoupled;
    CR_CHECK(c->adj_lam.alloc(4 * (size_t)n));
    CR_CHECK(c->adj_qbar.alloc(9 * (size_t)n));
    // mu's cotangent, lambda . NABI and Q per outlet; then the blocks' partial sums of the former
    const int gi = grid_for(4LL * c->nelem, 128, kAdjBlocksPerSM), ge = grid_for(c->nelem, 128, kAdjBlocksPerSM);
    const int gf = c->nface > 0 ? grid_for(c->nface, 128, 4) : 0;
    const int nscal = 1 + 2 * nc, npart = gi + ge + gf;
    CR_CHECK(c->adj_scal.alloc((size_t)nscal + npart));
    double* mupart = c->adj_scal.p + nscal;
    launch(k_adj_mask, grid_for(n, 256), 256, 0, s, (const int*)c->iBC.p, d_lam, c->adj_lam.p, n);
    const AdjConst C = make_adj_consts();
    AdjParams P;
    P.rho = p.rho;
    P.Dtgl = p.Dtgl;
    P.dtsfct = p.dtsfct;
    P.taucfct = p.taucfct;
    P.stabflux = p.stabflux_coeff;
    P.idiff = p.idiff;
    const double4* x4 = c->x.p;
    const double4* y4 = reinterpret_cast<const double4*>(d_y);
    const double4* a4 = reinterpret_cast<const double4*>(d_ac);
    const double4* l4 = reinterpret_cast<const double4*>(c->adj_lam.p);
    const int gn = grid_for((long long)kAdjLanes * n, 256);
    launch(k_adj_interior, gi, 128, 0, s, (const int4*)c->ien.p, x4, y4, a4, (const double*)c->qres.p, l4, c->nelem, C, P,
           p.mu, c->erec.p, mupart);
    int np = gi;
    if (p.idiff == 1) {
        launch(k_adj_qnode, gn, 256, 0, s, (const int*)c->diag.p, (const int*)c->soff.p, (const int*)c->slist.p,
               (const double*)c->erec.p, (const double*)c->rmass.p, n, c->adj_qbar.p);
        launch(k_adj_asiq, ge, 128, 0, s, (const int4*)c->ien.p, x4, y4, (const double*)c->adj_qbar.p, c->nelem, C, p.mu,
               c->qrec.p, mupart + np);
        np += ge;
    }
    launch(k_adj_node, gn, 256, 0, s, (const int*)c->diag.p, (const int*)c->soff.p, (const int*)c->slist.p,
           (const double*)c->erec.p, p.idiff == 1 ? (const double*)c->qrec.p : nullptr, n, d_ybar,
           d_abar);
    if (c->nface > 0) {
        launch(k_adj_faces, gf, 128, 0, s, (const int4*)c->ienb.p, (const int*)c->iBCB.p, x4, y4, l4,
                c->nface, C, P, p.mu, d_ybar, mupart + np);
        np += gf;
    }
    launch(k_adj_sum, 1, 256, 0, s, (const double*)mupart, np, c->adj_scal.p);
    if (nc > 0) {
        const int* doff = c->d_onode_off.p;
        double* sl = c->adj_scal.p + 1;        // s_k = lambda . NABI
        double* qf = c->adj_scal.p + 1 + nc;   // Q_k = y . NABI
        launch(k_adj_flow, nc, 256, 0, s, (const int*)c->onodes.p, doff, (const double4*)c->onabi.p, l4, sl);
        launch(k_adj_flow, nc, 256, 0, s, (const int*)c->onodes.p, doff, (const double4*)c->onabi.p, y4, qf);
        // coef1 as the primal residual put it on the device
        launch(k_adj_pvsq, dim3(8, nc), 256, 0, s, (const int*)c->onodes.p, doff, (const double4*)c->onabi.p,
               (const double*)sl, (const double*)c->coefs.p, nc, d_ybar);
    }
    std::vector<double> hs((size_t)nscal, 0.0);
    CR_CUDA(cudaMemcpyAsync(hs.data(), c->adj_scal.p, sizeof(double) * nscal, cudaMemcpyDeviceToHost, s));
    CR_CUDA(cudaStreamSynchronize(s));
    CR_CUDA(cudaGetLastError());
    if (mubar) *mubar = hs[0];
    for (int k = 0; k < nc; ++k) {
        // p_k = -(Q_k coef1_k) - coef2_k; res(vel) += p_k NABI
        if (c1bar) c1bar[k] = -hs[1 + nc + k] * hs[1 + k];
        if (c2bar) c2bar[k] = -hs[1 + k];
    }
    return CRIMSON_OK;
}

}  // namespace crimson
