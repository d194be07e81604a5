// rt_fine.cu — finest-level matrix-free hex8 operator on the dense node box.
//
// Restates (on a dense x-fastest box instead of GS-ordered index tables):
//   update_residual_OTFA_{NS,WS}_kernel  grid/Grid.cu:1450-1557
//   applyK_OTFA_kernel                   grid/Grid.cu:2439-2517
//   gs_relax_OTFA_{NS,WS}_kernel         grid/Grid.cu:792-1066
//   computeSensitivity_kernel            optimization/optimization.cu:44-107
// Node v gathers rho_e^p * KE[(7-i) block row] * u_e over its 8 incident
// elements i (element offset (i%2-1, i/2%2-1, i/4-1)); with supports, fixed
// neighbours contribute u = 0 and fixed rows are identity (applyK), zero
// (residual) or n_e * I (GS).
#include <cuda_runtime.h>

#include <algorithm>

#include "rt_element.cuh"
#include "rt_internal.h"

namespace {

constexpr int FINE_BS = 256;

// the 3 x 21 couplings of an element's vertex 0 to its other vertices (KE rows 0..2); the other vertices' follow by
// reflection: KE[v][v ^ m][r][c] = s_r s_c KE[0][m][r][c], s_t = -1 where v has bit t, else 1
template <typename T>
struct VertexRow {
    T k[7][3][3];
    T diag_a, diag_b;  // KE[v][v] = a I + b (s s^T - I)
};

// x / d from id = 1 / d: the product's remainder added back, which rounds as the division does (Markstein)
template <typename T>
__device__ __forceinline__ T quotient(T x, T d, T id) {
    const T q = x * id;
    return fma(fma(-d, q, x), id, q);
}

// diag: the common diagonal entry of the node's block, off: its entries xy, xz, yz
template <typename T>
__device__ __forceinline__ void block_gs(T diag, const T (&off)[3], const T (&F)[3], const T (&KU)[3], T (&uu)[3],
                                         bool backward) {
    const T id = T(1) / diag;  // off the chain of the three updates
    if (!backward) {
        uu[0] = quotient(F[0] - off[0] * uu[1] - off[1] * uu[2] - KU[0], diag, id);
        uu[1] = quotient(F[1] - off[0] * uu[0] - off[2] * uu[2] - KU[1], diag, id);
        uu[2] = quotient(F[2] - off[1] * uu[0] - off[2] * uu[1] - KU[2], diag, id);
    } else {
        uu[2] = quotient(F[2] - off[1] * uu[0] - off[2] * uu[1] - KU[2], diag, id);
        uu[1] = quotient(F[1] - off[0] * uu[0] - off[2] * uu[2] - KU[1], diag, id);
        uu[0] = quotient(F[0] - off[0] * uu[1] - off[1] * uu[2] - KU[0], diag, id);
    }
}

// x with its sign bit flipped where mask has bit 31
__device__ __forceinline__ double flip_sign(double x, unsigned mask) {
    return __hiloint2double((int)((unsigned)__double2hiint(x) ^ mask), __double2loint(x));
}
__device__ __forceinline__ float flip_sign(float x, unsigned mask) {
    return __uint_as_float(__float_as_uint(x) ^ mask);
}

// one colour of the 8-colour point-block GS; colour c = x%2 + 2(y%2) + 4(z%2).  4 lanes per node (lane = 8 * quadrant +
// node, 8 nodes of a row per warp), each with the two elements of its (y, z) quadrant: a colour of a small grid has too
// few nodes to fill the GPU with a thread each, and the two elements share a face, so that a lane loads 11 neighbours
// where two lanes with an element each load 14.  A warp's load touches 4 rows; with 8 lanes per node, one per element,
// it touched 8, and the L1's wavefronts were the bound.  The loads depend on the box alone, not on the weights, which
// only select.  With the reflected vertex row the products take their matrix entries from the kernel parameters,
// whichever vertex the node is.
// FP64, per colour with the launch: 64x32x32 10.7 us with 8 lanes, 9.8 with 4; 128x48x40 19.0, 13.9; 65x41x33 without
// supports 12.5, 8.9.  Blocks per SM: without supports the compiler keeps all 33 loads in flight and spills at 4 blocks
// (10.7 us); with them 3 blocks take 16.2 us on 128x48x40.
constexpr int GS_BS = 128;

template <typename T, bool WS>
__global__ void __launch_bounds__(GS_BS, WS ? 4 : 3) k_fine_gs(int nx, int ny, int nz, int color, bool backward,
                                                       const uint8_t* __restrict__ code, const float* __restrict__ w,
                                                       const VertexRow<T> kr, T* __restrict__ u,
                                                       const T* __restrict__ f) {
    const int vx = nx + 1, vy = ny + 1, vz = nz + 1;
    const long plane = (long)vx * vy, nv = plane * vz;
    const int px = color & 1, py = (color >> 1) & 1, pz = (color >> 2) & 1;
    const unsigned cx = (vx - px + 1) / 2, cy = (vy - py + 1) / 2, cz = (vz - pz + 1) / 2;
    const unsigned nc = cx * cy * cz;
    const int lane = threadIdx.x & 31, quad = lane >> 3;
    const int dy = quad & 1 ? 1 : -1, dz = quad & 2 ? 1 : -1;  // the quadrant's side of the node
    const unsigned my = dy < 0 ? 0x80000000u : 0u, mz = dz < 0 ? 0x80000000u : 0u;
    const unsigned stride = gridDim.x * (GS_BS / 4);
    for (unsigned t0 = blockIdx.x * (GS_BS / 4) + (threadIdx.x >> 5) * 8; t0 < nc; t0 += stride) {
        const unsigned t = t0 + (lane & 7);
        T KU[3] = {T(0), T(0), T(0)}, F[3] = {T(0), T(0), T(0)}, uu[3] = {T(0), T(0), T(0)};
        T sw = T(0), swx = T(0);  // sums of the two weights, and with the sign of x
        uint32_t cd = 0;
        long v = 0;
        if (t < nc) {
            const int x = px + 2 * (int)(t % cx), y = py + 2 * (int)(t / cx % cy), z = pz + 2 * (int)(t / (cx * cy));
            v = x + (long)vx * y + plane * z;
            if (quad == 0) {
                cd = code[v];
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    F[c] = f[c * nv + v];
                    uu[c] = u[c * nv + v];
                }
            }
            const int ey = y + (dy - 1) / 2, ez = z + (dz - 1) / 2;
            if (ey >= 0 && ez >= 0 && ey < ny && ez < nz) {
                const float* we = w + x + (long)nx * (ey + (long)ny * ez);
                const bool in[2] = {x > 0, x < nx};
                const float wv[2] = {in[0] ? we[-1] : 0.f, in[1] ? we[0] : 0.f};
                // rows of KE in the vertex's reflected frame (sx u0, sy u1, sz u2); the shared nodes' u0 apart, whose sign
                // depends on the side
                T sh0[3] = {}, sh[3] = {}, p[2][3] = {};
                // vertex m of the node's elements on side d; nodes without an element, and fixed ones, count as zero
                auto vertex = [&](int m, int d, bool load, bool use, T (&acc0)[3], T (&acc)[3]) {
                    const long n = v + (m & 1 ? 2 * d - 1 : 0) + (m & 2 ? dy * (long)vx : 0) + (m & 4 ? dz * plane : 0);
                    T un[3] = {T(0), T(0), T(0)};
                    if (load) {
                        if (WS) use = use && code[n] <= 1;
#pragma unroll
                        for (int c = 0; c < 3; c++) un[c] = u[c * nv + n];
                    }
#pragma unroll
                    for (int c = 0; c < 3; c++) un[c] = use ? un[c] : T(0);
                    if (d == 0 && (m & 1)) un[0] = -un[0];
                    un[1] = flip_sign(un[1], my);
                    un[2] = flip_sign(un[2], mz);
#pragma unroll
                    for (int r = 0; r < 3; r++) {
                        acc0[r] += kr.k[m - 1][r][0] * un[0];
                        acc[r] += kr.k[m - 1][r][1] * un[1];
                        acc[r] += kr.k[m - 1][r][2] * un[2];
                    }
                };
#pragma unroll
                for (int m = 2; m < 8; m += 2) vertex(m, 0, true, wv[0] != 0.f || wv[1] != 0.f, sh0, sh);
#pragma unroll
                for (int d = 0; d < 2; d++)
#pragma unroll
                    for (int m = 1; m < 8; m += 2) vertex(m, d, in[d], wv[d] != 0.f, p[d], p[d]);
                const T w0 = T(wv[0]), w1 = T(wv[1]);
                sw = w0 + w1;
                swx = w1 - w0;
                KU[0] = w1 * (p[1][0] + (sh[0] + sh0[0])) - w0 * (p[0][0] + (sh[0] - sh0[0]));
                KU[1] = flip_sign(w1 * (p[1][1] + (sh[1] + sh0[1])) + w0 * (p[0][1] + (sh[1] - sh0[1])), my);
                KU[2] = flip_sign(w1 * (p[1][2] + (sh[2] + sh0[2])) + w0 * (p[0][2] + (sh[2] - sh0[2])), mz);
            }
        }
        // sums of w, w sx sy, w sx sz, w sy sz
        T S[4] = {sw, flip_sign(swx, my), flip_sign(swx, mz), flip_sign(sw, my ^ mz)};
#pragma unroll
        for (int o = 8; o < 32; o <<= 1) {
#pragma unroll
            for (int c = 0; c < 3; c++) KU[c] += __shfl_xor_sync(0xffffffffu, KU[c], o);
#pragma unroll
            for (int c = 0; c < 4; c++) S[c] += __shfl_xor_sync(0xffffffffu, S[c], o);
        }
        if (quad != 0 || cd == 0) continue;
        if (WS && cd > 1u) {  // n_e u = f
#pragma unroll
            for (int c = 0; c < 3; c++) uu[c] = F[c] / T(cd >> 2);
        } else {
            const T off[3] = {kr.diag_b * S[1], kr.diag_b * S[2], kr.diag_b * S[3]};
            block_gs(kr.diag_a * S[0], off, F, KU, uu, backward);
        }
        u[v] = uu[0]; u[nv + v] = uu[1]; u[2 * nv + v] = uu[2];
    }
}

// four elements per thread (the arrays are allocations of their own).  255x256x128, with the launch: 49 us with one,
// 38 us here, powf bound
__global__ void k_penalty(long ne, const uint8_t* __restrict__ eact, const float* __restrict__ rho, float p,
                          float* __restrict__ w) {
    const long n4 = ne / 4, tid = blockIdx.x * (long)blockDim.x + threadIdx.x;
    for (long i = tid; i < n4; i += (long)gridDim.x * blockDim.x) {
        const uchar4 a = reinterpret_cast<const uchar4*>(eact)[i];
        const float4 r = reinterpret_cast<const float4*>(rho)[i];
        reinterpret_cast<float4*>(w)[i] = make_float4(a.x ? powf(r.x, p) : 0.f, a.y ? powf(r.y, p) : 0.f,
                                                      a.z ? powf(r.z, p) : 0.f, a.w ? powf(r.w, p) : 0.f);
    }
    if (tid < ne - 4 * n4) {
        const long e = 4 * n4 + tid;
        w[e] = eact[e] ? powf(rho[e], p) : 0.f;
    }
}

// ELEM_C = false: s_e = -p rho^(p-1) u_e.KE u_e (computeSensitivity_kernel, optimization/optimization.cu:44-107);
// ELEM_C = true: c_e = rho^p u_e.KE u_e (elementCompliance_kernel, grid/Grid.cu:3434-3480).
// u_e.KE u_e = h.Kt h with h = H u_e the Hadamard transform of the element's displacements (rt_element.cuh): 45
// products instead of 576.  A thread marches an element column through a z-chunk and keeps the x and y stages of the
// node layer below, 48 adds and 12 loads per element, issued a layer ahead.  255x256x128: 835 us with the dense 24 x 24
// product, 288 us with one chain of 45 products and the loads in their own layer, 167 us here.  Latency bound, at three
// blocks per SM (four, with spills: 197 us).
template <bool ELEM_C>
__global__ void __launch_bounds__(128) k_sensitivity(int nx, int ny, int nz, int zchunk, const uint8_t* __restrict__ eact,
                                                     const float* __restrict__ rho, float p,
                                                     const rte::KtVals<double> kt, const double* __restrict__ u,
                                                     float* __restrict__ sens) {
    const int x = blockIdx.x * 32 + (threadIdx.x & 31), y = blockIdx.y * 4 + (threadIdx.x >> 5);
    if (x >= nx || y >= ny) return;
    const int vx = nx + 1, vy = ny + 1;
    const long plane = (long)vx * vy, nv = plane * (nz + 1);
    const int Z0 = blockIdx.z * zchunk, Z1 = min(Z0 + zchunk, nz);
    long v = x + (long)vx * y + plane * Z0, e = x + (long)nx * (y + (long)ny * Z0);
    double raw[12];  // the four nodes of the next layer, loaded a layer ahead
    float nro = 0.f;
    bool nact = false;
    auto load = [&](long n) {
#pragma unroll
        for (int c = 0; c < 3; c++) {
            const double* q = u + c * nv + n;
            raw[4 * c] = q[0];
            raw[4 * c + 1] = q[1];
            raw[4 * c + 2] = q[vx];
            raw[4 * c + 3] = q[vx + 1];
        }
    };
    // x and y stages of the four nodes of a layer: index 3 (mx + 2 my) + component
    auto face = [&](double (&F)[12]) {
#pragma unroll
        for (int c = 0; c < 3; c++) {
            const double a = raw[4 * c], b = raw[4 * c + 1], d = raw[4 * c + 2], g = raw[4 * c + 3];
            F[c] = (a + b) + (d + g);
            F[3 + c] = (a - b) + (d - g);
            F[6 + c] = (a + b) - (d + g);
            F[9 + c] = (a - b) - (d - g);
        }
    };
    double lo[12], hi[12];
    load(v);
    face(lo);
    load(v + plane);
    nact = eact[e];
    nro = rho[e];
    for (int z = Z0; z < Z1; z++, e += (long)nx * ny) {
        v += plane;
        face(hi);
        const bool act = nact;
        const float ro = nro;
        if (z + 1 < Z1) {
            load(v + plane);
            nact = eact[e + (long)nx * ny];
            nro = rho[e + (long)nx * ny];
        }
        double h[24];
#pragma unroll
        for (int q = 0; q < 12; q++) {
            h[q] = lo[q] + hi[q];
            h[12 + q] = lo[q] - hi[q];
            lo[q] = hi[q];
        }
        // row sums first: 66 products instead of 90, in short chains instead of one of 45
        double zz[24], t[3] = {0.0, 0.0, 0.0};
#pragma unroll
        for (int k = 0; k < 45; k++) {
            if (k == 0 || rte::KT_R[k - 1] != rte::KT_R[k]) zz[rte::KT_R[k]] = kt.v[k] * h[rte::KT_C[k]];
            else zz[rte::KT_R[k]] += kt.v[k] * h[rte::KT_C[k]];
        }
#pragma unroll
        for (int r = 3; r < 24; r++) t[r % 3] += h[r] * zz[r];
        // u.KE u >= 0: where an element moves rigidly, the rounding left over may be negative
        const double s = fabs(t[0] + t[1] + t[2]);
        if (ELEM_C)
            sens[e] = act ? (float)(s * (double)powf(ro, p)) : 0.f;
        else
            sens[e] = act ? (float)(-s * (double)(p * powf(ro, p - 1.f))) : 0.f;
    }
}

unsigned fine_grid(rt_ctx* c, long n) {
    long b = rt_blocks(n, FINE_BS);
    long cap = (long)c->sm_count * 16;
    return (unsigned)(b < cap ? b : cap);
}

}  // namespace

namespace rtk {

int penalty_weights(rt_hier* h) {
    rt_level& L = h->L[0];
    return rt_launch(h->ctx, "penalty_weights", [&] {
        k_penalty<<<fine_grid(h->ctx, (L.ne + 3) / 4), FINE_BS, 0, h->ctx->stream>>>(L.ne, L.eact, h->rho, h->P.power_penalty,
                                                                          h->w);
    });
}

template <typename T>
int fine_gs(rt_hier* h, T* u, const T* f, bool backward) {
    rt_level& L = h->L[0];
    const char* nm = sizeof(T) == 8 ? "fine_gs_f64" : "fine_gs_f32";
    VertexRow<T> kr;
    for (int m = 1; m < 8; m++)
        for (int r = 0; r < 3; r++)
            for (int c = 0; c < 3; c++) kr.k[m - 1][r][c] = (T)h->KE[r * 24 + 3 * m + c];
    kr.diag_a = (T)h->KE[0];
    kr.diag_b = (T)h->KE[1];
    for (int cc = 0; cc < 8; cc++) {
        int col = backward ? 7 - cc : cc;
        long ncol = (long)((L.vx - (col & 1) + 1) / 2) * ((L.vy - ((col >> 1) & 1) + 1) / 2) *
                    ((L.vz - ((col >> 2) & 1) + 1) / 2);
        if (ncol == 0) continue;
        RT_CHECK(rt_launch(h->ctx, nm, [&] {
            const unsigned g = (unsigned)std::min<long>((4 * ncol + GS_BS - 1) / GS_BS, (long)h->ctx->sm_count * 64);
            if (h->has_support)
                k_fine_gs<T, true><<<g, GS_BS, 0, h->ctx->stream>>>(L.nx, L.ny, L.nz, col, backward, h->ncode, h->w,
                                                                      kr, u, f);
            else
                k_fine_gs<T, false><<<g, GS_BS, 0, h->ctx->stream>>>(L.nx, L.ny, L.nz, col, backward, h->ncode, h->w,
                                                                       kr, u, f);
        }));
    }
    return RT_OK;
}

template <bool ELEM_C>
static int sens_launch(rt_hier* h, const char* name, const double* u, float* out) {
    rt_level& L = h->L[0];
    const int bx = (L.nx + 31) / 32, by = (L.ny + 3) / 4;
    int zc = 16;  // 1/16 of the node layers read twice; shorter chunks where blocks are few
    while (zc > 2 && (long)bx * by * ((L.nz + zc - 1) / zc) < 8L * h->ctx->sm_count) zc /= 2;
    const rte::KtVals<double> kt = rte::make_kt<double>(h);
    return rt_launch(h->ctx, name, [&] {
        k_sensitivity<ELEM_C><<<dim3(bx, by, (L.nz + zc - 1) / zc), 128, 0, h->ctx->stream>>>(
            L.nx, L.ny, L.nz, zc, L.eact, h->rho, h->P.power_penalty, kt, u, out);
    });
}

int sensitivity(rt_hier* h, const double* u) { return sens_launch<false>(h, "sensitivity", u, h->sens); }

int element_compliance(rt_hier* h, const double* u, float* out) {
    return sens_launch<true>(h, "element_compliance", u, out);
}

template int fine_gs<double>(rt_hier*, double*, const double*, bool);
template int fine_gs<float>(rt_hier*, float*, const float*, bool);

}  // namespace rtk
