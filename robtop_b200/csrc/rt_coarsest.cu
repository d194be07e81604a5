// rt_coarsest.cu — coarsest-level direct solve on the device.
//
// The reference downloads the coarsest stencil, builds a dense matrix and
// factors it on the host with Eigen::BDCSVD (Grid::buildCoarsestSystem,
// grid/Grid.cpp:1884-1939), then does a D2H / svd.solve / H2D round trip every
// V-cycle (Grid::solve_fem_host, grid/Grid.cpp:1981-2043).  Here the dense
// matrix is assembled, inverted (blocked Gauss-Jordan, one cooperative launch with a
// grid barrier per 32 pivots) and applied (GEMV) without leaving the GPU.
// Without supports the matrix is singular with the rigid modes as null space;
// the minimum-norm solve of BDCSVD is reproduced as A^+ = (A + a R R^T)^-1 - R R^T / a.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <cmath>
#include <vector>

#include "rt_internal.h"

namespace cg = cooperative_groups;

namespace {

__global__ void k_assemble_dense(int vx, int vy, int vz, long nv, int na, const int* __restrict__ aidx,
                                 const int* __restrict__ rowof, const double* __restrict__ st, double* __restrict__ A) {
    const int n = 3 * na;
    const long tot = (long)na * 27 * 9;
    for (long t = blockIdx.x * (long)blockDim.x + threadIdx.x; t < tot; t += (long)gridDim.x * blockDim.x) {
        const int i = (int)(t / 243), q = (int)(t % 243), k = q / 9, rc = q % 9;
        const int v = aidx[i];
        const int x = v % vx, y = (v / vx) % vy, z = v / (vx * vy);
        const int jx = x + k % 3 - 1, jy = y + (k / 3) % 3 - 1, jz = z + k / 9 - 1;
        if (jx < 0 || jy < 0 || jz < 0 || jx >= vx || jy >= vy || jz >= vz) continue;
        const int j = rowof[jx + vx * (jy + vy * jz)];
        if (j < 0) continue;
        A[(long)(3 * i + rc / 3) * n + 3 * j + rc % 3] = st[(long)q * nv + v];
    }
}

__global__ void k_trace(int n, const double* __restrict__ A, double* __restrict__ out) {
    __shared__ double sh[256];
    double s = 0;
    for (int i = threadIdx.x; i < n; i += blockDim.x) s += A[(long)i * n + i];
    sh[threadIdx.x] = s;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) {
        if (threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) out[0] = sh[0] / n;
}

// In-place blocked Gauss-Jordan inversion of an SPD matrix (no pivoting needed), one grid barrier per GJ_B columns.
// With the step's panels C = A(:, K), R = A(K, :) as they were and P = A(K, K)^-1, every tile is independent:
//   A(i, j) -= (C_i P) R_j,  A(K, j) = P R_j,  A(i, K) = -C_i P,  A(K, K) = P.
// Every block inverts the 32 x 32 pivot block itself (cheaper than a second barrier), takes strips of one tile row,
// so that C_i P is formed once per strip, and writes the parts of the next step's panels that it updated into the
// other pair of panel buffers.  status[0] != 0 reports a non-positive pivot.  n = 1260: a barrier and a pass over
// the matrix per column took 14.6 ms, 1.36 ms here.
constexpr int GJ_B = 32, GJ_T = 256;

__global__ void __launch_bounds__(GJ_T) k_gauss_jordan(int n, double* __restrict__ A, double* __restrict__ panels,
                                                       int* __restrict__ status) {
    cg::grid_group grid = cg::this_grid();
    __shared__ double P[GJ_B][GJ_B + 1], Ct[GJ_B][GJ_B + 1], W[GJ_B][GJ_B + 1], Rt[GJ_B][GJ_B];
    __shared__ int bad;
    const int tid = threadIdx.x, lane = tid & 31, wr = (tid >> 5) * 4;  // a thread's column and first of its 4 rows
    const int nb = (n + GJ_B - 1) / GJ_B;
    const long pn = (long)n * GJ_B;  // one panel: C [n][32], R [32][n]
    const int strips = (int)gridDim.x / nb > 0 ? (int)gridDim.x / nb : 1;  // per tile row
    const int per = (nb + strips - 1) / strips;                           // tiles of a strip
    const int items = nb * strips;
    for (long t = blockIdx.x * (long)GJ_T + tid; t < pn; t += (long)gridDim.x * GJ_T) {
        const int i = (int)(t / GJ_B), k = (int)(t % GJ_B);
        panels[t] = k < n ? A[(long)i * n + k] : 0.0;
        panels[pn + t] = t / n < n ? A[t] : 0.0;  // rows 0..31
    }
    grid.sync();
    for (int kb = 0; kb < nb; kb++) {
        const double *C = panels + 2 * pn * (kb & 1), *R = C + pn;
        double *Cn = panels + 2 * pn * ((kb + 1) & 1), *Rn = Cn + pn;
        const int k0 = kb * GJ_B, kw = min(GJ_B, n - k0);
        // P = inverse of the pivot block (the identity past the matrix's end)
        for (int i = tid; i < GJ_B * GJ_B; i += GJ_T) {
            const int r = i / GJ_B, c = i % GJ_B;
            P[r][c] = r < kw && c < kw ? C[(long)(k0 + r) * GJ_B + c] : (r == c ? 1.0 : 0.0);
        }
        if (tid == 0) bad = 0;
        __syncthreads();
        for (int k = 0; k < kw; k++) {
            const double pv = P[k][k];
            double row = P[k][lane], col[4];
#pragma unroll
            for (int q = 0; q < 4; q++) col[q] = P[wr + q][k];
            if (!(pv > 0)) {
                if (tid == 0) bad = k0 + k + 1;
                break;  // uniform: every thread of every block reads the same pivot
            }
            const double ip = 1.0 / pv;
            row *= ip;
            __syncthreads();
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const int r = wr + q;
                if (r == k) P[r][lane] = lane == k ? ip : row;
                else P[r][lane] = lane == k ? -col[q] * ip : P[r][lane] - col[q] * row;
            }
            __syncthreads();
        }
        __syncthreads();
        if (bad != 0) {
            if (blockIdx.x == 0 && tid == 0) status[0] = bad;
            return;
        }
        for (int it = blockIdx.x; it < items; it += gridDim.x) {
            const int ib = it / strips, j0 = (it - ib * strips) * per, j1 = min(j0 + per, nb);
            const int i0 = ib * GJ_B;
            if (j0 >= j1) continue;
            __syncthreads();
            if (ib == kb) {  // this tile row becomes P R_j
                for (int i = tid; i < GJ_B * GJ_B; i += GJ_T) W[i / GJ_B][i % GJ_B] = P[i / GJ_B][i % GJ_B];
            } else {  // W = C_i P
                for (int i = tid; i < GJ_B * GJ_B; i += GJ_T) {
                    const int r = i / GJ_B, c = i % GJ_B;
                    Ct[r][c] = i0 + r < n && c < kw ? C[(long)(i0 + r) * GJ_B + c] : 0.0;
                }
                __syncthreads();
                double w[4] = {0, 0, 0, 0};
                for (int k = 0; k < GJ_B; k++) {
                    const double b = P[k][lane];
#pragma unroll
                    for (int q = 0; q < 4; q++) w[q] += Ct[wr + q][k] * b;
                }
#pragma unroll
                for (int q = 0; q < 4; q++) W[wr + q][lane] = w[q];
            }
            for (int jb = j0; jb < j1; jb++) {
                const int j = jb * GJ_B + lane;
                __syncthreads();
                for (int i = tid; i < GJ_B * GJ_B; i += GJ_T) {
                    const int r = i / GJ_B, c = i % GJ_B;
                    Rt[r][c] = r < kw && jb * GJ_B + c < n ? R[(long)r * n + jb * GJ_B + c] : 0.0;
                }
                double a[4], s[4] = {0, 0, 0, 0};
#pragma unroll
                for (int q = 0; q < 4; q++)
                    a[q] = ib != kb && jb != kb && i0 + wr + q < n && j < n ? A[(long)(i0 + wr + q) * n + j] : 0.0;
                __syncthreads();
                if (jb == kb) {
#pragma unroll
                    for (int q = 0; q < 4; q++) s[q] = W[wr + q][lane];
                } else {
                    for (int k = 0; k < GJ_B; k++) {
                        const double b = Rt[k][lane];
#pragma unroll
                        for (int q = 0; q < 4; q++) s[q] += W[wr + q][k] * b;
                    }
                }
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    const int i = i0 + wr + q;
                    if (i >= n || j >= n) continue;
                    const double v = ib == kb ? s[q] : a[q] - s[q];
                    A[(long)i * n + j] = v;
                    if (jb == kb + 1) Cn[(long)i * GJ_B + lane] = v;
                    if (ib == kb + 1) Rn[(long)(wr + q) * n + j] = v;
                }
            }
        }
        grid.sync();
    }
}

__global__ void k_sub_rrt(int n, int nr, const double* __restrict__ R, const double* __restrict__ alpha,
                          double* __restrict__ A) {
    const double ia = 1.0 / alpha[0];
    for (long t = blockIdx.x * (long)blockDim.x + threadIdx.x; t < (long)n * n; t += (long)gridDim.x * blockDim.x) {
        const int i = (int)(t / n), j = (int)(t % n);
        double s = 0;
        for (int a = 0; a < nr; a++) s += R[(long)a * n + i] * R[(long)a * n + j];
        A[t] -= s * ia;
    }
}

__global__ void k_add_rrt_dev(int n, int nr, const double* __restrict__ R, const double* __restrict__ alpha,
                              double* __restrict__ A) {
    const double a = alpha[0];
    for (long t = blockIdx.x * (long)blockDim.x + threadIdx.x; t < (long)n * n; t += (long)gridDim.x * blockDim.x) {
        const int i = (int)(t / n), j = (int)(t % n);
        double s = 0;
        for (int q = 0; q < nr; q++) s += R[(long)q * n + i] * R[(long)q * n + j];
        A[t] += a * s;
    }
}

template <typename TI, typename TO>
__global__ void k_gather_active(int na, long nv, const int* __restrict__ aidx, const TI* __restrict__ f,
                                TO* __restrict__ d) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < na; i += gridDim.x * blockDim.x) {
        const int v = aidx[i];
        d[3 * i] = (TO)f[v]; d[3 * i + 1] = (TO)f[nv + v]; d[3 * i + 2] = (TO)f[2 * nv + v];
    }
}

// u = Ainv d, one warp per row, scattered back to the node box (u zeroed first by the caller)
template <typename T, typename TU>
__global__ void k_gemv_scatter(int na, long nv, const int* __restrict__ aidx, const T* __restrict__ Ainv,
                               const T* __restrict__ d, TU* __restrict__ u) {
    const int n = 3 * na;
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    for (int i = warp; i < n; i += nwarps) {
        T s = 0;
        const T* row = Ainv + (long)i * n;
        for (int j = lane; j < n; j += 32) s += row[j] * d[j];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
        if (lane == 0) u[(long)(i % 3) * nv + aidx[i / 3]] = (TU)s;
    }
}

// the coarsest solve in one launch, n <= CS_MAXN: every block gathers the right-hand side of the active nodes into
// shared memory, a warp multiplies a row of the inverse (8 loads in flight per lane), and the inactive nodes are set to
// zero.  The V-cycle visits it up to 8 times per iteration; gather, memset and product took three launches.  n = 1260:
// 14.7 us with the launch.
constexpr int CS_MAXN = 4096;
template <typename T>
__global__ void __launch_bounds__(256) k_coarsest(int na, int nv, const int* __restrict__ aidx,
                                                  const uint8_t* __restrict__ vact, const double* __restrict__ Ainv,
                                                  const T* __restrict__ f, T* __restrict__ u) {
    extern __shared__ double d[];
    const int n = 3 * na, lane = threadIdx.x & 31;
    for (int i = threadIdx.x; i < na; i += 256) {
        const int v = aidx[i];
        d[3 * i] = (double)f[v];
        d[3 * i + 1] = (double)f[nv + v];
        d[3 * i + 2] = (double)f[2 * nv + v];
    }
    for (int v = blockIdx.x * 256 + threadIdx.x; v < nv; v += gridDim.x * 256)
        if (!vact[v]) u[v] = u[nv + v] = u[2 * nv + v] = T(0);
    __syncthreads();
    for (int i = blockIdx.x * 8 + (threadIdx.x >> 5); i < n; i += gridDim.x * 8) {
        const double* row = Ainv + (long)i * n;
        double s[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        for (int j0 = lane; j0 < n; j0 += 256) {
            double a[8];
#pragma unroll
            for (int q = 0; q < 8; q++) a[q] = j0 + 32 * q < n ? row[j0 + 32 * q] : 0.0;
#pragma unroll
            for (int q = 0; q < 8; q++)
                if (j0 + 32 * q < n) s[q] += a[q] * d[j0 + 32 * q];
        }
        double t = ((s[0] + s[1]) + (s[2] + s[3])) + ((s[4] + s[5]) + (s[6] + s[7]));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
        if (lane == 0) u[(i % 3) * nv + aidx[i / 3]] = (T)t;
    }
}

}  // namespace

namespace rtk {

// what the coarsest set-up needs besides the matrix, made once per hierarchy: the stream-ordered allocations and the
// host round trip of the index map that every call made here took 1 ms and, where the pool had given its memory back
// to the system, up to a second
static int coarsest_workspace(rt_hier* h, bool rigid) {
    rt_ctx* c = h->ctx;
    rt_level& L = h->L.back();
    const int na = L.na, n = 3 * na;
    if (L.crow && (L.crigid || !rigid)) return RT_OK;
    std::vector<int> aidx_h(na), rowof_h(L.nv, -1);
    RT_CUDA(c, cudaMemcpyAsync(aidx_h.data(), L.aidx, sizeof(int) * na, cudaMemcpyDeviceToHost, c->stream));
    RT_CUDA(c, cudaStreamSynchronize(c->stream));
    for (int i = 0; i < na; i++) rowof_h[aidx_h[i]] = i;
    if (!L.cpanels) RT_CUDA(c, cudaMalloc(&L.cpanels, sizeof(double) * 4 * GJ_B * n));
    if (!L.cstatus) RT_CUDA(c, cudaMalloc(&L.cstatus, sizeof(int)));
    if (!L.crow) {
        RT_CUDA(c, cudaMalloc(&L.crow, sizeof(int) * L.nv));
        RT_CUDA(c, cudaMemcpyAsync(L.crow, rowof_h.data(), sizeof(int) * L.nv, cudaMemcpyHostToDevice, c->stream));
        RT_CUDA(c, cudaStreamSynchronize(c->stream));
    }
    if (rigid && !L.crigid) {
        // orthonormal rigid modes at the coarsest active nodes (positions are static)
        std::vector<double> Rh((size_t)6 * n, 0.0);
        for (int i = 0; i < na; i++) {
            int v = aidx_h[i];
            double p[3] = {(double)(v % L.vx), (double)((v / L.vx) % L.vy), (double)(v / (L.vx * L.vy))};
            double ph[3][3] = {{0, -p[2], p[1]}, {p[2], 0, -p[0]}, {-p[1], p[0], 0}};
            for (int t = 0; t < 3; t++) Rh[(size_t)t * n + 3 * i + t] = 1.0;
            for (int k = 0; k < 3; k++)
                for (int t = 0; t < 3; t++) Rh[(size_t)(3 + k) * n + 3 * i + t] = ph[t][k];
        }
        for (int a = 0; a < 6; a++) {
            for (int b = 0; b < a; b++) {
                double d = 0;
                for (int q = 0; q < n; q++) d += Rh[(size_t)a * n + q] * Rh[(size_t)b * n + q];
                for (int q = 0; q < n; q++) Rh[(size_t)a * n + q] -= d * Rh[(size_t)b * n + q];
            }
            double nn = 0;
            for (int q = 0; q < n; q++) nn += Rh[(size_t)a * n + q] * Rh[(size_t)a * n + q];
            nn = std::sqrt(nn);
            for (int q = 0; q < n; q++) Rh[(size_t)a * n + q] /= nn;
        }
        RT_CUDA(c, cudaMalloc(&L.crigid, sizeof(double) * 6 * n));
        RT_CUDA(c, cudaMemcpyAsync(L.crigid, Rh.data(), sizeof(double) * 6 * n, cudaMemcpyHostToDevice, c->stream));
        RT_CUDA(c, cudaStreamSynchronize(c->stream));
    }
    return RT_OK;
}

int coarsest_setup(rt_hier* h) {
    rt_ctx* c = h->ctx;
    rt_level& L = h->L.back();
    const int na = L.na, n = 3 * na;
    if (na == 0) return rt_fail(c, RT_ESTATE, "coarsest level has no active node");
    const bool no_support = (h->P.mode == RT_MODE_NSCF || h->P.mode == RT_MODE_NSFF);
    RT_CHECK(coarsest_workspace(h, no_support));
    const int* rowof = L.crow;
    double *panels = L.cpanels, *R = L.crigid;
    int* status = L.cstatus;
    RT_CUDA(c, cudaMemsetAsync(status, 0, sizeof(int), c->stream));
    RT_CUDA(c, cudaMemsetAsync(L.ainv, 0, sizeof(double) * (size_t)n * n, c->stream));
    RT_CHECK(rt_launch(c, "coarsest_assemble", [&] {
        long tot = (long)na * 243;
        unsigned g = (unsigned)std::min<long>((tot + 255) / 256, (long)c->sm_count * 8);
        k_assemble_dense<<<g, 256, 0, c->stream>>>(L.vx, L.vy, L.vz, L.nv, na, L.aidx, rowof, L.st, L.ainv);
    }));
    unsigned gnn = (unsigned)std::min<long>(((long)n * n + 255) / 256, (long)c->sm_count * 8);
    if (no_support) {
        RT_CHECK(rt_launch(c, "coarsest_trace", [&] { k_trace<<<1, 256, 0, c->stream>>>(n, L.ainv, h->scal + 60); }));
        RT_CHECK(rt_launch(c, "coarsest_add_rrt",
                           [&] { k_add_rrt_dev<<<gnn, 256, 0, c->stream>>>(n, 6, R, h->scal + 60, L.ainv); }));
    }
    // cooperative Gauss-Jordan
    int dev = c->device, nb_per_sm = 0;
    RT_CUDA(c, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb_per_sm, k_gauss_jordan, GJ_T, 0));
    int coop = 0;
    RT_CUDA(c, cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev));
    if (!coop || nb_per_sm < 1) return rt_fail(c, RT_ECUDA, "cooperative launch unavailable");
    const long tiles = (long)((n + GJ_B - 1) / GJ_B) * ((n + GJ_B - 1) / GJ_B);
    const unsigned gblocks = (unsigned)std::min<long>((long)c->sm_count * std::min(nb_per_sm, 2), tiles);
    double* Aptr = L.ainv;
    int nn_ = n;
    void* args[] = {&nn_, &Aptr, &panels, &status};
    RT_CHECK(rt_launch(c, "coarsest_gauss_jordan", [&] {
        cudaLaunchCooperativeKernel((void*)k_gauss_jordan, gblocks, GJ_T, args, 0, c->stream);
    }));
    if (no_support) {
        RT_CHECK(rt_launch(c, "coarsest_sub_rrt",
                           [&] { k_sub_rrt<<<gnn, 256, 0, c->stream>>>(n, 6, R, h->scal + 60, L.ainv); }));
    }
    int st_h = 0;
    RT_CUDA(c, cudaMemcpyAsync(&st_h, status, sizeof(int), cudaMemcpyDeviceToHost, c->stream));
    RT_CUDA(c, cudaStreamSynchronize(c->stream));
    if (st_h != 0) return rt_fail(c, RT_ENAN, "coarsest matrix not positive definite (pivot %d)", st_h - 1);
    return RT_OK;
}

// u = A^-1 f on the coarsest level.  The inverse and the product are FP64 in both precisions
// of the V-cycle: the coarse operator's conditioning (the stiffness contrast survives the
// averaging) would amplify the rounding of an FP32 copy of the inverse.
template <typename T>
int coarsest_solve(rt_hier* h, const T* f, T* u) {
    rt_ctx* c = h->ctx;
    rt_level& L = h->L.back();
    if (3 * L.na <= CS_MAXN)
        return rt_launch(c, sizeof(T) == 8 ? "coarsest_solve_f64" : "coarsest_solve_f32", [&] {
            const unsigned g = (unsigned)std::min<long>((3L * L.na + 7) / 8, (long)c->sm_count * 4);
            k_coarsest<T><<<g, 256, sizeof(double) * 3 * L.na, c->stream>>>(L.na, (int)L.nv, L.aidx, L.vact, L.ainv, f, u);
        });
    RT_CHECK(rt_launch(c, sizeof(T) == 8 ? "coarsest_gather_f64" : "coarsest_gather_f32", [&] {
        k_gather_active<T, double><<<(L.na + 255) / 256, 256, 0, c->stream>>>(L.na, L.nv, L.aidx, f, L.dvec);
    }));
    RT_CUDA(c, cudaMemsetAsync(u, 0, sizeof(T) * 3 * L.nv, c->stream));
    const int n = 3 * L.na;
    return rt_launch(c, sizeof(T) == 8 ? "coarsest_gemv_f64" : "coarsest_gemv_f32", [&] {
        unsigned g = (unsigned)std::min<long>(((long)n * 32 + 255) / 256, (long)c->sm_count * 8);
        k_gemv_scatter<double, T><<<g, 256, 0, c->stream>>>(L.na, L.nv, L.aidx, L.ainv, L.dvec, u);
    });
}

template int coarsest_solve<double>(rt_hier*, const double*, double*);
template int coarsest_solve<float>(rt_hier*, const float*, float*);

}  // namespace rtk
