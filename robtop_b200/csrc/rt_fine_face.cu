// rt_fine_face.cu — finest-level operator marching element columns through z, with the transforms of the
// element vectors shared between neighbours and their partial results carried in registers.
//
// Same operators as rt_fine_tile.cu (residual, applyK, damped block Jacobi, Chebyshev step;
// grid/Grid.cu:1450-1557, 2439-2517).  The operator has few flops per byte, but the tile kernels spend
// ~880 thread-instructions per node on it (24 shared loads, 24 shared stores and two full 24-point butterflies
// per element, 24 shared loads per node), and the issue slots bound them, at a third of the HBM rate.  Here:
//
//  * The 8-vertex Hadamard transform (KE = T Kt T^T / 64, see rt_element.cuh) is done one axis at a time.  The
//    x stage of an edge serves 4 elements, the y stage of a face 2 (the element below keeps it in registers for
//    the element above), only the z stage is per element: 6 + 12 + 24 adds instead of 72, and the same on the
//    way back, where neighbours' results are added between the stages, so that no scatter remains.
//  * A lane owns element column X0 - 1 + lane and node column X0 - 1 + lane, a warp one element row.  x neighbours
//    meet by shuffles; the upper edge of a warp's row goes to the next warp, 6 values (in FP64 smoothing 2 weight sums
//    as well) per lane and layer through shared memory, with one barrier per layer.  Lanes 1..30 finish nodes; a block
//    of W warps finishes 30 x (W - 1) nodes per layer.
//  * The loads of the next layer and of this layer's output stage are issued before the arithmetic (FP32 Chebyshev on
//    511x256x256, when it formed the diagonal block itself: 874 us with them behind it, 666).
//  * FP64 K u, with 12 warps per SM, waits longest at the barrier: there a warp arrives at an mbarrier when its edge of
//    layer t is written, and waits (with a limit) before the output of layer t, which follows the x stage and the loads
//    of layer t + 1 (511x256x256: 897 us with __syncthreads, 766 us).  The other forms hold the inputs of the output
//    stage as well and got slower with it (FP64 residual 850, 938 us with it; FP32 residual 490, 600 us).
//  * Two element rows per warp, with the edge between them in registers, need 128 registers in FP32: that Chebyshev
//    step 736 us.
//  * The 3x3 diagonal block of a node needs four signed sums of its 8 weights, factorised the same way.  FP64 steps form
//    and invert it; FP32 steps read the inverse that k_fine_dinv made in FP64.  Inverted in FP32 here, a step from zero
//    had 2 to 3 times the error, and entries past 1e12 or below 1e-13 left FP32's range in the determinant (511x256x256,
//    z-chunk 16: Jacobi 637 us so, 715 us read; Chebyshev 686, 715 us); formed here in FP64 it needs registers that are
//    not there (Jacobi 682 us, Chebyshev 928 us; 773 us with 20 warps per SM instead of 24).
//
// Fixed and inactive nodes enter the element products as zero (the reference's WS rule); out[] follows
// rt_fine_tile.cu's rules for them.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>

#include "rt_element.cuh"
#include "rt_internal.h"
#include "rt_tc.cuh"

namespace {

constexpr int FACE_NX = 30;  // node columns a warp finishes (lanes 1..30)

// warps per block: FP64 12, one block per SM (registers), 8 for the smoothing steps (two blocks of 8 with spills:
// residual 1287 us, Chebyshev 2431 us on 511x256x256); FP32 8, three blocks
constexpr int face_warps(bool f64, int mode) { return f64 && mode < 2 ? 12 : 8; }

// 1 / det of a node's block; 0 where all its elements have zero weight (the node keeps its value)
__device__ __forceinline__ double block_rcp(double det, double sw) { return sw == 0.0 ? 0.0 : 1.0 / det; }

// a fixed node's rule f / n_e, from its code; 0 without a weighted element
template <typename T>
__device__ __forceinline__ T fixed_value(T f, uint32_t code) {
    return code >> 2 ? f / T(code >> 2) : T(0);
}

// the grid's sum of x in out[0]: block sums, added by the last block to finish in their order (the ticket counter is
// left at zero); W warps per block
template <int W>
__device__ __forceinline__ void face_grid_sum(double x, double* __restrict__ partials, double* __restrict__ out,
                                              unsigned* __restrict__ ticket) {
    __shared__ double sd[W];
    __shared__ bool last;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    auto block_sum = [&](double v) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
        __syncthreads();
        if (lane == 0) sd[w] = v;
        __syncthreads();
        double a = 0;
#pragma unroll
        for (int i = 0; i < W; i++) a += sd[i];
        return a;
    };
    const double b = block_sum(x);
    const unsigned nb = gridDim.x * gridDim.y * gridDim.z;
    if (threadIdx.x == 0) {
        partials[blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z)] = b;
        __threadfence();
        last = atomicInc(ticket, nb - 1) == nb - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    double a = 0;
    for (unsigned i = threadIdx.x; i < nb; i += 32 * W) a += __ldcg(partials + i);
    a = block_sum(a);
    if (threadIdx.x == 0) out[0] = a;
}

// MODE 0: r = f - K u (fixed rows: r = f)     MODE 1: out = K u (fixed rows: u)
// MODE 2: unew = u + omega D^-1 (f - K u)     MODE 3: Chebyshev step kstep: d = a_k d + b_k D^-1 (f - K u), unew = u + d
// (fixed nodes in MODE 2/3: unew = f / n_e, d = 0; inactive nodes: 0; nodes whose elements all have zero weight: D^-1 and
// f / n_e count as 0, as with the stored blocks)
// code: per node, bit 0 active, bit 1 fixed (supports), for fixed nodes n_e << 2
template <typename T, bool WS, int MODE, int W, int MINB, bool DOT>
__global__ void __launch_bounds__(32 * W, MINB)
    k_fine_face(int nx, int ny, int nz, int zchunk, const uint8_t* __restrict__ code, const float* __restrict__ wgt,
                const rte::KtVals<T> kt, const T* __restrict__ dinv, const T* __restrict__ u, const T* __restrict__ f,
                T* __restrict__ out, T omega, T* __restrict__ dvec, const double* __restrict__ coef, int kstep, double* __restrict__ partials,
                double* __restrict__ dot_out, unsigned* __restrict__ ticket, double* __restrict__ err) {
    constexpr bool STORED = sizeof(T) == 4 && MODE >= 2, BLOCK = sizeof(T) == 8 && MODE >= 2;  // inverse blocks read, formed
    constexpr int NX = BLOCK ? 8 : 6;  // values handed to the next warp
    constexpr bool LATE = sizeof(T) == 8 && MODE == 1;
    __shared__ T S[2][W][NX][32];
    __shared__ uint64_t bar;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    T cheb_a = T(0), cheb_b = T(0);
    if (MODE == 3) {
        cheb_a = (T)coef[2 * kstep];
        cheb_b = (T)coef[2 * kstep + 1];
    }
    const int vx = nx + 1, vy = ny + 1, vz = nz + 1;
    const int nv = vx * vy * vz, plane = vx * vy, eplane = nx * ny;  // 3 nv < 2^31 (launch_face checks)
    const int ci = blockIdx.x * FACE_NX - 1 + lane;
    const int ri = blockIdx.y * (W - 1) - 1 + w;  // the warp's element row = first node row
    const int Z0 = blockIdx.z * zchunk, Z1 = min(Z0 + zchunk, vz);
    const bool c_ok = ci >= 0 && ci < vx, n_ok[2] = {c_ok && ri >= 0 && ri < vy, c_ok && ri + 1 >= 0 && ri + 1 < vy};
    const bool e_ok = ci >= 0 && ci < nx && ri >= 0 && ri < ny;
    const bool own = lane >= 1 && lane <= FACE_NX && n_ok[0] && w > 0;  // the lane finishes node (ci, ri)
    if (LATE) {
        if (threadIdx.x == 0) {
            rttc::mbar_init(&bar, W);
            rttc::fence_mbar_init();
        }
        __syncthreads();
    }

    T pu[2][3];      // u of the next node layer, as stored
    uint32_t pc[2];  // its node codes
    float pw;        // weight of the element layer below it
    // node layer L (index vn of the lane's first node) and element layer L - 1 (index en)
    auto fetch = [&](int L, int vn, int en) {
        const bool zn = L >= 0 && L < vz, ze = L >= 1 && L <= nz;
#pragma unroll
        for (int r = 0; r < 2; r++) {
            const int v = vn + r * vx;
            pc[r] = 0;
            if (zn && n_ok[r]) {
                pc[r] = code[v];
                pu[r][0] = u[v];
                pu[r][1] = u[nv + v];
                pu[r][2] = u[2 * nv + v];
            }
        }
        pw = ze && e_ok ? wgt[en] : 0.f;
    };
    // x stage of a node row: sums and differences along the edge to the next column (active free nodes only)
    auto x_stage = [&](const T (&p)[3], uint32_t c, T (&E)[6]) {
#pragma unroll
        for (int q = 0; q < 3; q++) {
            const T un = c == 1u ? p[q] : T(0);
            const T nb = __shfl_down_sync(0xffffffffu, un, 1);
            E[q] = un + nb;
            E[3 + q] = un - nb;
        }
    };

    double pq = 0;  // DOT: the thread's part of u . out
    T F[12];        // forward face data of node layer t
    T G[12];        // inverse z output of element layer t - 1 toward node layer t
    uint32_t cc = 0, co = 0;              // node codes of the next layer and of the output stage's layer
    T Qp[4] = {T(0), T(0), T(0), T(0)};   // signed weight sums of the element layer below the output stage's layer
    T X[6], wa = T(0), wb = T(0);         // the output stage's x-edge data and weight sums along x
    T fv[3], dv[3], uo[3], inv[6];        // its inputs
    int vn = ci + vx * ri + plane * (Z0 - 1);  // node (ci, ri) of layer t
    int en = ci + nx * ri + eplane * (Z0 - 1);
    fetch(Z0 - 1, vn, en - eplane);
    {
        T E0[6], E1[6];
        x_stage(pu[0], pc[0], E0);
        x_stage(pu[1], pc[1], E1);
#pragma unroll
        for (int q = 0; q < 6; q++) {
            F[q] = E0[q] + E1[q];
            F[6 + q] = E0[q] - E1[q];
        }
#pragma unroll
        for (int q = 0; q < 12; q++) G[q] = T(0);
    }
    fetch(Z0, vn + plane, en);

    uint32_t phase = 0;
    // node layer t (index v of the lane's node) from X, once every warp has written its edge of it.  The other buffer of
    // S is written next; this one again only after the barrier of that one
    auto output = [&](int t, int v) {
        if (!LATE) {
            __syncthreads();
        } else {
            if (!rttc::mbar_wait(&bar, phase)) {  // not reached: all warps of a block arrive in every layer
                *err = 4.0;
#pragma unroll
                for (int q = 0; q < 6; q++) X[q] = T(NAN);  // in the layer's nodes and u . out, which a solve reports
                pq = NAN;
            }
            phase ^= 1;
        }
        T wa_b = T(0), wb_b = T(0);
        if (w > 0) {
#pragma unroll
            for (int q = 0; q < 6; q++) X[q] += S[t & 1][w - 1][q][lane];
            if (BLOCK) {
                wa_b = S[t & 1][w - 1][NX - 2][lane];
                wb_b = S[t & 1][w - 1][NX - 1][lane];
            }
        }
        T acc[3];
#pragma unroll
        for (int c = 0; c < 3; c++) acc[c] = X[c] + X[3 + c] + __shfl_up_sync(0xffffffffu, X[c] - X[3 + c], 1);
        T Q[4];
        if (BLOCK) {
            Q[0] = wa + wa_b;  // sum w
            Q[1] = wb - wb_b;  // sum w sx sy
            Q[2] = wa - wa_b;  // sum w sy
            Q[3] = wb + wb_b;  // sum w sx
        }
        if (t >= Z0 && own) {
            const bool act = co != 0, fixed = WS && co > 1u;
            T o[3] = {T(0), T(0), T(0)}, dn[3] = {T(0), T(0), T(0)};
            if (MODE == 0) {
#pragma unroll
                for (int c = 0; c < 3; c++) o[c] = act ? (fixed ? fv[c] : fv[c] - acc[c]) : T(0);
            } else if (MODE == 1) {
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    o[c] = act ? (fixed ? uo[c] : acc[c]) : T(0);
                    if (DOT) pq += (double)uo[c] * (double)o[c];
                }
            } else if (fixed) {
#pragma unroll
                for (int c = 0; c < 3; c++) o[c] = fixed_value(fv[c], co);
            } else if (act) {
                T rr[3], zz[3];
#pragma unroll
                for (int c = 0; c < 3; c++) rr[c] = fv[c] - acc[c];
                if constexpr (STORED) {
                    zz[0] = inv[0] * rr[0] + inv[1] * rr[1] + inv[2] * rr[2];
                    zz[1] = inv[1] * rr[0] + inv[3] * rr[1] + inv[4] * rr[2];
                    zz[2] = inv[2] * rr[0] + inv[4] * rr[1] + inv[5] * rr[2];
                } else {
                    const T sw = Q[0] + Qp[0], sxy = Q[1] + Qp[1], sxz = Q[3] - Qp[3], syz = Q[2] - Qp[2];
                    const T A = kt.diag_a * sw, bxy = kt.diag_b * sxy, bxz = kt.diag_b * sxz, byz = kt.diag_b * syz;
                    // inverse of [[A,bxy,bxz],[bxy,A,byz],[bxz,byz,A]]
                    const T c00 = A * A - byz * byz, c01 = byz * bxz - bxy * A, c02 = bxy * byz - A * bxz;
                    const T c11 = A * A - bxz * bxz, c12 = bxy * bxz - A * byz, c22 = A * A - bxy * bxy;
                    const T id = block_rcp(A * c00 + bxy * c01 + bxz * c02, sw);
                    zz[0] = id * (c00 * rr[0] + c01 * rr[1] + c02 * rr[2]);
                    zz[1] = id * (c01 * rr[0] + c11 * rr[1] + c12 * rr[2]);
                    zz[2] = id * (c02 * rr[0] + c12 * rr[1] + c22 * rr[2]);
                }
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    if (MODE == 2) {
                        o[c] = uo[c] + omega * zz[c];
                    } else {
                        dn[c] = cheb_a * dv[c] + cheb_b * zz[c];  // dv = 0 in step 0
                        o[c] = uo[c] + dn[c];
                    }
                }
            }
#pragma unroll
            for (int c = 0; c < 3; c++) out[c * nv + v] = o[c];
            if (MODE == 3)
#pragma unroll
                for (int c = 0; c < 3; c++) dvec[c * nv + v] = dn[c];
        }
        if (BLOCK)
#pragma unroll
            for (int q = 0; q < 4; q++) Qp[q] = Q[q];
    };

    for (int t = Z0 - 1;; t++, vn += plane, en += eplane) {
        if (!LATE && t == Z1) break;
        // ---- node layer t + 1 into the x stage, then the loads of layer t + 2
        T E0[6], E1[6], wv = T(0);
        uint32_t cn = 0;
        if (!LATE || t < Z1) {
            x_stage(pu[0], pc[0], E0);
            x_stage(pu[1], pc[1], E1);
            cn = pc[0];
            wv = (T)pw;
            if (t + 1 < Z1) fetch(t + 2, vn + 2 * plane, en + eplane);
        }
        if (LATE) {
            if (t >= Z0) output(t - 1, vn - plane);
            if (t == Z1) break;
        }
        co = cc;
        cc = cn;
        // inputs of layer t's output stage (u is in L1: the layer was fetched two layers ago)
        const bool ld = t >= Z0 && own && co != 0;
#pragma unroll
        for (int c = 0; c < 3; c++) {
            fv[c] = (MODE != 1 && ld) ? f[c * nv + vn] : T(0);
            dv[c] = (MODE == 3 && ld && kstep > 0) ? dvec[c * nv + vn] : T(0);
            uo[c] = ((MODE >= 2 || DOT || (WS && MODE == 1 && co > 1u)) && ld) ? u[c * nv + vn] : T(0);
        }
        if (STORED)
#pragma unroll
            for (int q = 0; q < 6; q++) inv[q] = ld ? dinv[q * (long)nv + vn] : T(0);
        // ---- element layer t
        if (BLOCK) {
            const T wl = __shfl_up_sync(0xffffffffu, wv, 1);
            wa = wv + wl;
            wb = wv - wl;
        }
        T h[24], z[24], Ft[12];
#pragma unroll
        for (int q = 0; q < 12; q++) {
            const T hi = q < 6 ? E0[q] + E1[q] : E0[q - 6] - E1[q - 6];
            h[q] = F[q] + hi;
            h[12 + q] = F[q] - hi;
            F[q] = hi;
        }
        // rows 0..2 of Kt (the rigid translations) are empty; a row's first product initialises it
#pragma unroll
        for (int k = 0; k < 45; k++) {
            if (k == 0 || rte::KT_R[k - 1] != rte::KT_R[k]) z[rte::KT_R[k]] = kt.v[k] * h[rte::KT_C[k]];
            else z[rte::KT_R[k]] += kt.v[k] * h[rte::KT_C[k]];
        }
#pragma unroll
        for (int q = 0; q < 12; q++) {
            const T s = q < 3 ? z[12 + q] : z[q] + z[12 + q], d = q < 3 ? -z[12 + q] : z[q] - z[12 + q];
            Ft[q] = G[q] + wv * s;  // toward node layer t, with element layer t - 1's part
            G[q] = wv * d;          // toward node layer t + 1
        }
#pragma unroll
        for (int q = 0; q < 6; q++) {
            X[q] = Ft[q] + Ft[6 + q];
            S[t & 1][w][q][lane] = Ft[q] - Ft[6 + q];
        }
        if (BLOCK) {
            S[t & 1][w][NX - 2][lane] = wa;
            S[t & 1][w][NX - 1][lane] = wb;
        }
        if (LATE) {
            __syncwarp();
            if (lane == 0) rttc::mbar_arrive(&bar);
        }
        if (!LATE) output(t, vn);
    }
    // no second launch and no second read of u and out for p.q
    if (DOT) face_grid_sum<W>(pq, partials, dot_out, ticket);
}

// The smoothing step from u = 0, where K u needs no evaluation: out = omega D^-1 f (MODE 2) or out = d = b_0 D^-1 f
// (MODE 3), fixed nodes f / n_e (d = 0).  A thread marches one node column through a z-chunk with the weight sums of
// the element layer below, the block in FP64; 29 B (MODE 2) or 41 B per node in FP32, the full step moves 90.
// FP32 Chebyshev, 511x256x256: 343 us with the block in FP32, 404 us so.
template <typename T, int MODE, bool DOT>
__global__ void __launch_bounds__(256) k_fine_diag(int nx, int ny, int nz, int zchunk, const uint8_t* __restrict__ code,
                                                   const float* __restrict__ wgt, double diag_a, double diag_b,
                                                   const T* __restrict__ f, T* __restrict__ out, T omega,
                                                   T* __restrict__ dvec, const double* __restrict__ coef,
                                                   double* __restrict__ partials, double* __restrict__ dot_out,
                                                   unsigned* __restrict__ ticket) {
    double fo = 0;  // DOT: the thread's part of f . out
    const int vx = nx + 1, vy = ny + 1, vz = nz + 1;
    const int x = blockIdx.x * 32 + (threadIdx.x & 31), y = blockIdx.y * 8 + (threadIdx.x >> 5);
    const bool col_ok = x < vx && y < vy;
    if (!DOT && !col_ok) return;
    const T scale = MODE == 3 ? (T)coef[1] : omega;
    const int Z0 = blockIdx.z * zchunk, Z1 = col_ok ? min(Z0 + zchunk, vz) : 0;
    const long plane = (long)vx * vy, nv = plane * vz, eplane = (long)nx * ny;
    const long col = x + (long)vx * y, ecol = x + (long)nx * y;
    const bool x0 = x > 0, x1 = x < nx, y0 = y > 0, y1 = y < ny;
    double Qp[4] = {0, 0, 0, 0};
#pragma unroll 2
    for (int t = Z0 - 1; t < Z1; t++) {
        double w00 = 0, w10 = 0, w01 = 0, w11 = 0;  // element (x - 1 + i, y - 1 + j) of layer t
        if (t >= 0 && t < nz) {
            const float* we = wgt + ecol + eplane * t;
            if (x0 && y0) w00 = we[-1 - nx];
            if (x1 && y0) w10 = we[-nx];
            if (x0 && y1) w01 = we[-1];
            if (x1 && y1) w11 = we[0];
        }
        const double a0 = w10 + w00, b0 = w10 - w00, a1 = w11 + w01, b1 = w11 - w01;
        const double Q[4] = {a1 + a0, b1 - b0, a1 - a0, b1 + b0};  // sums of w, w sx sy, w sy, w sx
        if (t >= Z0) {
            const long v = col + plane * t;
            const uint32_t c = code[v];
            const T f0 = f[v], f1 = f[nv + v], f2 = f[2 * nv + v];
            T o[3] = {T(0), T(0), T(0)};
            if (c == 1u) {
                const double sw = Q[0] + Qp[0], sxy = Q[1] + Qp[1], sxz = Q[3] - Qp[3], syz = Q[2] - Qp[2];
                const double A = diag_a * sw, bxy = diag_b * sxy, bxz = diag_b * sxz, byz = diag_b * syz;
                const double c00 = A * A - byz * byz, c01 = byz * bxz - bxy * A, c02 = bxy * byz - A * bxz;
                const double c11 = A * A - bxz * bxz, c12 = bxy * bxz - A * byz, c22 = A * A - bxy * bxy;
                const double id = block_rcp(A * c00 + bxy * c01 + bxz * c02, sw) * scale;
                o[0] = (T)(id * (c00 * f0 + c01 * f1 + c02 * f2));
                o[1] = (T)(id * (c01 * f0 + c11 * f1 + c12 * f2));
                o[2] = (T)(id * (c02 * f0 + c12 * f1 + c22 * f2));
            } else if (c > 1u) {
                o[0] = fixed_value(f0, c);
                o[1] = fixed_value(f1, c);
                o[2] = fixed_value(f2, c);
            }
#pragma unroll
            for (int q = 0; q < 3; q++) {
                out[q * nv + v] = o[q];
                if (MODE == 3) dvec[q * nv + v] = c == 1u ? o[q] : T(0);
            }
            if (DOT) fo += (double)f0 * (double)o[0] + (double)f1 * (double)o[1] + (double)f2 * (double)o[2];
        }
#pragma unroll
        for (int q = 0; q < 4; q++) Qp[q] = Q[q];
    }
    if (DOT) face_grid_sum<8>(fo, partials, dot_out, ticket);
}

// The same step from the stored inverse blocks, FP32 only: 53 B (MODE 2) or 65 B per node, but no sums and no division,
// and two nodes' loads in flight per thread.  Chebyshev, with the launch, against k_fine_diag: 97x61x45 10.7 us (14.7),
// 255x256x128 96 us (135), 511x256x256 358 us (404); with one node per trip 11.3, 119 and 422 us.
constexpr int DIAG_U = 2;

template <int MODE>
__global__ void __launch_bounds__(256) k_fine_diag_stored(long nv, const uint8_t* __restrict__ code,
                                                          const float* __restrict__ dinv, const float* __restrict__ f,
                                                          float* __restrict__ out, float omega, float* __restrict__ dvec,
                                                          const double* __restrict__ coef) {
    const float scale = MODE == 3 ? (float)coef[1] : omega;
    const long st = gridDim.x * 256L;
    for (long v0 = blockIdx.x * 256L + threadIdx.x; v0 < nv; v0 += DIAG_U * st) {
        uint32_t c[DIAG_U];
        float inv[DIAG_U][6], r[DIAG_U][3];
#pragma unroll
        for (int k = 0; k < DIAG_U; k++) {
            const long v = v0 + k * st;
            c[k] = 0;
            if (v >= nv) break;
            c[k] = code[v];
#pragma unroll
            for (int q = 0; q < 6; q++) inv[k][q] = dinv[q * nv + v];
#pragma unroll
            for (int q = 0; q < 3; q++) r[k][q] = f[q * nv + v];
        }
#pragma unroll
        for (int k = 0; k < DIAG_U; k++) {
            const long v = v0 + k * st;
            if (v >= nv) break;
            float o[3] = {0.f, 0.f, 0.f};
            if (c[k] == 1u) {
                o[0] = scale * (inv[k][0] * r[k][0] + inv[k][1] * r[k][1] + inv[k][2] * r[k][2]);
                o[1] = scale * (inv[k][1] * r[k][0] + inv[k][3] * r[k][1] + inv[k][4] * r[k][2]);
                o[2] = scale * (inv[k][2] * r[k][0] + inv[k][4] * r[k][1] + inv[k][5] * r[k][2]);
            } else if (c[k] > 1u) {
#pragma unroll
                for (int q = 0; q < 3; q++) o[q] = fixed_value(r[k][q], c[k]);
            }
#pragma unroll
            for (int q = 0; q < 3; q++) {
                out[q * nv + v] = o[q];
                if (MODE == 3) dvec[q * nv + v] = c[k] == 1u ? o[q] : 0.f;
            }
        }
    }
}

// node codes read by k_fine_face: bit 0 active, bit 1 fixed, bits 2.. the number of elements of non-zero weight
// around a fixed node (its smoothing rule f / n_e).  Four nodes per thread (the arrays are allocations of their own):
// 255x256x128, with the launch: 37 us with one, 17 us here
__global__ void k_node_code(int nx, int ny, int nz, const uint8_t* __restrict__ vact, const uint8_t* __restrict__ vfix,
                            const float* __restrict__ w, uint8_t* __restrict__ code) {
    const int vx = nx + 1, vy = ny + 1;
    const long nv = (long)vx * vy * (nz + 1), n4 = nv / 4, tid = blockIdx.x * (long)blockDim.x + threadIdx.x;
    auto node = [&](long v, bool act, bool fix) {
        uint8_t c = act ? 1 : 0;
        if (act && fix) {
            const int x = (int)(v % vx), y = (int)((v / vx) % vy), z = (int)(v / ((long)vx * vy));
            int ne = 0;
            for (int i = 0; i < 8; i++) {
                const int ex = x - 1 + (i & 1), ey = y - 1 + ((i >> 1) & 1), ez = z - 1 + (i >> 2);
                if (ex >= 0 && ey >= 0 && ez >= 0 && ex < nx && ey < ny && ez < nz &&
                    w[ex + (long)nx * (ey + (long)ny * ez)] != 0.f)
                    ne++;
            }
            c = (uint8_t)(3 | (ne << 2));
        }
        return c;
    };
    for (long i = tid; i < n4; i += (long)gridDim.x * blockDim.x) {
        const uchar4 a = reinterpret_cast<const uchar4*>(vact)[i];
        const uchar4 f = vfix != nullptr ? reinterpret_cast<const uchar4*>(vfix)[i] : make_uchar4(0, 0, 0, 0);
        reinterpret_cast<uchar4*>(code)[i] = make_uchar4(node(4 * i, a.x, f.x), node(4 * i + 1, a.y, f.y),
                                                         node(4 * i + 2, a.z, f.z), node(4 * i + 3, a.w, f.w));
    }
    if (tid < nv - 4 * n4) {
        const long v = 4 * n4 + tid;
        code[v] = node(v, vact[v], vfix != nullptr && vfix[v]);
    }
}

template <typename T, bool WS, int MODE, bool DOT>
int launch_face_dot(rt_hier* h, const T* u, const T* f, T* out, double omega, const char* name, T* dvec,
                    const double* coef, int kstep, double* dot_out) {
    constexpr int W = face_warps(sizeof(T) == 8, MODE), MINB = sizeof(T) == 8 ? 1 : 3;
    rt_level& L = h->L[0];
    if (sizeof(T) == 4 && MODE >= 2 && !h->dinv32)
        return rt_fail(h->ctx, RT_ESTATE, "%s: the diagonal blocks have not been made", name);
    const int zc = h->tune[sizeof(T) == 8 ? 1 : 0][MODE].zchunk;
    const dim3 grid((L.vx + FACE_NX - 1) / FACE_NX, (L.vy + W - 2) / (W - 1), (L.vz + zc - 1) / zc);
    const rte::KtVals<T> kt = rte::make_kt<T>(h);
    return rt_launch(h->ctx, name, [&] {
        k_fine_face<T, WS, MODE, W, MINB, DOT><<<grid, 32 * W, 0, h->ctx->stream>>>(
            L.nx, L.ny, L.nz, zc, h->ncode, h->w, kt, reinterpret_cast<const T*>(h->dinv32), u, f, out, (T)omega, dvec, coef, kstep, h->kpart, dot_out,
            reinterpret_cast<unsigned*>(h->scal + RT_SCAL_TICKET), h->scal + RT_SCAL_ERR);
    });
}

}  // namespace

namespace rtk {

int node_codes(rt_hier* h) {
    rt_level& L = h->L[0];
    return rt_launch(h->ctx, "node_codes", [&] {
        k_node_code<<<(unsigned)std::min<long>((L.nv + 1023) / 1024, (long)h->ctx->sm_count * 16), 256, 0,
                      h->ctx->stream>>>(L.nx, L.ny, L.nz, L.vact, h->has_support ? h->vfix : nullptr, h->w, h->ncode);
    });
}

// one smoothing step from u = 0: Jacobi (coef null) or the first Chebyshev step; dot_out (optional, Jacobi) f . out
template <typename T>
int fine_smooth0(rt_hier* h, const T* f, T* out, double omega, T* dvec, const double* coef, double* dot_out) {
    rt_level& L = h->L[0];
    if constexpr (sizeof(T) == 4) {
        // where the following steps read the stored blocks they are there, and current; 32 blocks per SM (16: 380 us)
        const int v = h->tune[0][coef ? 3 : 2].variant;
        if (v == 8 && h->dinv32 && !dot_out)
            return rt_launch(h->ctx, "fine_smooth0_f32", [&] {
                const unsigned g = (unsigned)std::min<long>((L.nv + 255) / 256, (long)h->ctx->sm_count * 32);
                cudaStream_t s = h->ctx->stream;
                if (coef)
                    k_fine_diag_stored<3><<<g, 256, 0, s>>>(L.nv, h->ncode, h->dinv32, f, out, 0.f, dvec, coef);
                else
                    k_fine_diag_stored<2><<<g, 256, 0, s>>>(L.nv, h->ncode, h->dinv32, f, out, (float)omega, nullptr, nullptr);
            });
    }
    int zc = 32;  // 1/32 of the weight layers read twice; shorter chunks where blocks are few
    const long xy = (long)((L.vx + 31) / 32) * ((L.vy + 7) / 8);
    while (zc > 4 && xy * ((L.vz + zc - 1) / zc) < 8L * h->ctx->sm_count) zc /= 2;
    const dim3 grid((L.vx + 31) / 32, (L.vy + 7) / 8, (L.vz + zc - 1) / zc);
    unsigned* ticket = reinterpret_cast<unsigned*>(h->scal + RT_SCAL_TICKET);
    return rt_launch(h->ctx, sizeof(T) == 8 ? "fine_smooth0_f64" : "fine_smooth0_f32", [&] {
        auto go = [&](auto kern, T om, T* d, const double* cf) {
            kern<<<grid, 256, 0, h->ctx->stream>>>(L.nx, L.ny, L.nz, zc, h->ncode, h->w, h->KE[0], h->KE[1], f, out,
                                                   om, d, cf, h->kpart, dot_out, ticket);
        };
        if (coef) go(k_fine_diag<T, 3, false>, T(0), dvec, coef);
        else if (dot_out) go(k_fine_diag<T, 2, true>, (T)omega, (T*)nullptr, (const double*)nullptr);
        else go(k_fine_diag<T, 2, false>, (T)omega, (T*)nullptr, (const double*)nullptr);
    });
}
template int fine_smooth0<double>(rt_hier*, const double*, double*, double, double*, const double*, double*);
template int fine_smooth0<float>(rt_hier*, const float*, float*, double, float*, const double*, double*);

template <typename T, bool WS, int MODE>
int launch_face(rt_hier* h, const T* u, const T* f, T* out, double omega, const char* name, T* dvec,
                const double* coef, int kstep) {
    return launch_face_dot<T, WS, MODE, false>(h, u, f, out, omega, name, dvec, coef, kstep, nullptr);
}

// partial sums of K u's dot product: one per block of the smallest launch shape (7 rows, one layer)
size_t face_dot_partials(int vx, int vy, int vz) {
    return (size_t)((vx + FACE_NX - 1) / FACE_NX) * ((vy + 6) / 7) * vz;
}

// out = K u and dot_dev = u . out
template <typename T>
int fine_applyK_dot(rt_hier* h, const T* u, T* out, double* dot_dev) {
    const rt_tile_cfg& tn = h->tune[sizeof(T) == 8 ? 1 : 0][1];
    const long n = 3 * h->L[0].nv;
    if (tn.variant != 8 || n >= (1L << 31)) {  // the other kernels leave the dot product to a pass of its own
        RT_CHECK(fine_applyK<T>(h, u, out));
        if constexpr (sizeof(T) == 8) return dot(h, n, u, out, dot_dev);
        else return dot32(h, n, u, out, dot_dev);
    }
    const char* nm = sizeof(T) == 8 ? "fine_applyK_f64" : "fine_applyK_f32";
    return h->has_support ? launch_face_dot<T, true, 1, true>(h, u, nullptr, out, 0.0, nm, nullptr, nullptr, 0, dot_dev)
                          : launch_face_dot<T, false, 1, true>(h, u, nullptr, out, 0.0, nm, nullptr, nullptr, 0, dot_dev);
}
template int fine_applyK_dot<double>(rt_hier*, const double*, double*, double*);
template int fine_applyK_dot<float>(rt_hier*, const float*, float*, double*);

// the launch shape used before rt_autotune ran: the z-chunk whose waves of blocks march through the fewest layers
// (a chunk of zc layers takes zc + 2 steps).  Against the best of 2, 4 .. 64 layers, timed warm on 64x32x32, 129x97x85,
// 255x256x128 and 511x256x256: FP32 at most 6 % slower.  FP64 at most 2 % on the first two, but 16 layers where 64 are 7
// to 10 % faster on the last, and on 255x256x128 8 layers for K u, 233 us, and the residual, 251 us, where 64 take 193
// and 213 us (rt_autotune finds them)
rt_tile_cfg face_default(rt_ctx* c, bool f64, int mode, int vx, int vy, int vz) {
    const int w = face_warps(f64, mode);
    const long slots = (long)c->sm_count * (f64 ? 1 : 3);
    const long xy = (long)((vx + FACE_NX - 1) / FACE_NX) * ((vy + w - 2) / (w - 1));
    rt_tile_cfg best{8, 1, 2};
    long cost = -1;
    for (int zc = 2; zc <= 64; zc *= 2) {
        const long waves = (xy * ((vz + zc - 1) / zc) + slots - 1) / slots, cz = waves * (zc + 2);
        if (cost < 0 || cz < cost) {
            cost = cz;
            best.zchunk = zc;
        }
    }
    return best;
}

#define RT_INST_FACE(T, WS, M) \
    template int launch_face<T, WS, M>(rt_hier*, const T*, const T*, T*, double, const char*, T*, const double*, int);
#define RT_INST_FACE_T(T)                                                                                          \
    RT_INST_FACE(T, false, 0) RT_INST_FACE(T, false, 1) RT_INST_FACE(T, false, 2) RT_INST_FACE(T, false, 3)        \
    RT_INST_FACE(T, true, 0) RT_INST_FACE(T, true, 1) RT_INST_FACE(T, true, 2) RT_INST_FACE(T, true, 3)
RT_INST_FACE_T(float)
RT_INST_FACE_T(double)

}  // namespace rtk
