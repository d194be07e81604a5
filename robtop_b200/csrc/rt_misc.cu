// rt_misc.cu — reductions, vector updates, load projection, filter, OC and
// occupancy set-up kernels.
//
// Restates:
//   block_dot/norm kernels, dot/norm, parallel_sum_d, parallel_maxabs   culib/lib.cuh:521-1137
//     (here: single-pass deterministic block partials + one fixed-order final
//      sum, result left on the device)
//   forceProject / getForceSupport / setForceSupport   optimization/projection.cu:165-369
//   displacementProject                                 optimization/projection.cpp:374-392
//   filterSensitivity_kernel                            grid/Grid.cu:2323-2409
//   trySensMultiplier_kernel                            optimization/optimization.cu:136-162
//   cubeGridSetSolidVertices_kernel / setSolidElementFromFineGrid_kernel  grid/Grid.cu:2555-2632
//   mark_surface_nodes_kernel                           grid/Grid.cu:2005-2039
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include "rt_internal.h"

namespace cg = cooperative_groups;

namespace {

constexpr int RB = 256;  // reduction block size
constexpr int XR_U = 4;  // grid strides per trip in the fused update + reduction kernels

unsigned gridN(rt_ctx* c, long n, int bs = 256) {
    long b = rt_blocks(n, bs);
    long cap = (long)c->sm_count * 16;
    return (unsigned)(b < 1 ? 1 : (b < cap ? b : cap));
}

struct RedOut {
    double* partials;  // one set per block
    double* out;
    unsigned* ticket;
};

// blocks of a reduction: 2 per SM, fewer for short vectors
unsigned red_grid(long n) { return (unsigned)(n < (long)RT_RED_BLOCKS * RB ? (n + RB - 1) / RB > 0 ? (n + RB - 1) / RB : 1 : RT_RED_BLOCKS); }

// block sums of v[0..NV) in thread 0
template <int NV>
__device__ __forceinline__ void block_reduce(double (&v)[NV]) {
    __shared__ double sh[NV][RB / 32];
    __syncthreads();
#pragma unroll
    for (int k = 0; k < NV; k++) {
        double x = v[k];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
        if ((threadIdx.x & 31) == 0) sh[k][threadIdx.x >> 5] = x;
    }
    __syncthreads();
    if (threadIdx.x < 32) {
#pragma unroll
        for (int k = 0; k < NV; k++) {
            double x = threadIdx.x < RB / 32 ? sh[k][threadIdx.x] : 0.0;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
            v[k] = x;
        }
    }
}

// the grid's sums of v[0..NV) in out: every block stores its own, and the last one to finish (a ticket counter, left
// at zero again) adds them in a fixed order, so that the sum does not depend on which block that is.  One launch
// where a second one added the partial sums, three times a PCG iteration.
template <int NV>
__device__ __forceinline__ bool grid_reduce(double (&v)[NV], const RedOut& o) {
    __shared__ bool last;
    block_reduce<NV>(v);
    if (threadIdx.x == 0) {
#pragma unroll
        for (int k = 0; k < NV; k++) o.partials[blockIdx.x * NV + k] = v[k];
        __threadfence();
        last = atomicInc(o.ticket, gridDim.x - 1) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return false;
    __threadfence();
    double t[NV];
#pragma unroll
    for (int k = 0; k < NV; k++) {
        t[k] = 0;
        for (int b = threadIdx.x; b < (int)gridDim.x; b += RB) t[k] += __ldcg(o.partials + (long)b * NV + k);
    }
    block_reduce<NV>(t);
    if (threadIdx.x == 0)
#pragma unroll
        for (int k = 0; k < NV; k++) o.out[k] = t[k];
    return true;  // in the block that holds the sums
}

__global__ void __launch_bounds__(RB) k_dot(long n, const double* __restrict__ a, const double* __restrict__ b,
                                            RedOut ro) {
    double v[1] = {0};
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) v[0] += a[i] * b[i];
    grid_reduce<1>(v, ro);
}

__global__ void k_axpy(long n, double a, const double* __restrict__ x, double* __restrict__ y) {
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) y[i] += a * x[i];
}

__global__ void k_f2d(long n, const float* __restrict__ a, double* __restrict__ b) {
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) b[i] = (double)a[i];
}

// b = float(a / s), s = sqrt(s_dev[0]) (scales the FP32 right-hand side to unit norm)
__global__ void k_d2f_scaled(long n, const double* __restrict__ a, float* __restrict__ b, const double* __restrict__ s) {
    const double inv = 1.0 / sqrt(fmax(s[0], 1e-300));
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x)
        b[i] = (float)(a[i] * inv);
}
__global__ void k_f2d_scaled(long n, const float* __restrict__ a, double* __restrict__ b, const double* __restrict__ s) {
    const double sc = sqrt(fmax(s[0], 1e-300));
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x)
        b[i] = (double)a[i] * sc;
}

// b += a * sqrt(s) (a coarse correction computed on a right-hand side scaled by 1 / sqrt(s))
__global__ void k_f2d_scaled_add(long n, const float* __restrict__ a, double* __restrict__ b,
                                 const double* __restrict__ s) {
    const double sc = sqrt(fmax(s[0], 1e-300));
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x)
        b[i] += (double)a[i] * sc;
}

// ---------------------------------------------------------------------------
// Vector passes of the PCG iteration, FP64 or FP32 vectors (T; dots summed in FP64).  z = sc * zs: the FP32 V-cycle's
// result is widened where it is used instead of being stored.  The flexible beta = (z.r - z.r_old) / rz_old is
// -(z.q) / (p.q), since r = r_old - alpha q with alpha = rz_old / (p.q), so no copy of the old residual is kept.  The
// step of x waits for the next iteration's pass over p (and one pass after the loop).  Per entry, FP64 vectors with
// an FP32 V-cycle: 84 bytes in 3 passes where 128 in 5 were moved (511x256x256: 2.2 -> 1.4 ms per iteration).
// scal: 10 z.r, 11 z.q, 12 the previous z.r, 20 p.q, 21 r.r, 24 the iteration.
// ---------------------------------------------------------------------------
template <typename TZ>
__device__ __forceinline__ double z_scale(const double* s) { return s ? sqrt(fmax(s[0], 1e-300)) : 1.0; }

// (z.r, z.q)
template <typename TZ, typename T>
__global__ void __launch_bounds__(RB) k_pcg_zdots(long n, const TZ* __restrict__ zs, const double* __restrict__ s,
                                                  const T* __restrict__ r, const T* __restrict__ q, RedOut ro) {
    const double sc = z_scale<TZ>(s);
    double v[2] = {0, 0};
    const long st = (long)gridDim.x * blockDim.x;
    for (long i0 = blockIdx.x * (long)blockDim.x + threadIdx.x; i0 < n; i0 += XR_U * st) {
        TZ a[XR_U];
        T ri[XR_U], qi[XR_U];
#pragma unroll
        for (int k = 0; k < XR_U; k++) {
            const long i = i0 + k * st;
            if (i < n) { a[k] = zs[i]; ri[k] = r[i]; qi[k] = q[i]; }
        }
#pragma unroll
        for (int k = 0; k < XR_U; k++) {
            if (i0 + k * st >= n) break;
            const double z = (double)a[k] * sc;
            v[0] += z * (double)ri[k];
            v[1] += z * (double)qi[k];
        }
    }
    grid_reduce<2>(v, ro);
}

// x += alpha p (the previous iteration's step), then p = z + beta p
template <typename TZ, typename T>
__global__ void __launch_bounds__(RB) k_pcg_xp(long n, const double* __restrict__ scal, const TZ* __restrict__ zs,
                                               const double* __restrict__ s, T* __restrict__ p, T* __restrict__ x) {
    const bool first = scal[24] == 0.0;
    const double sc = z_scale<TZ>(s), pq = scal[20];
    const T beta = first || pq == 0.0 ? T(0) : (T)(-scal[11] / pq), alpha = first || pq == 0.0 ? T(0) : (T)(scal[12] / pq);
    const long st = (long)gridDim.x * blockDim.x;
    for (long i0 = blockIdx.x * (long)blockDim.x + threadIdx.x; i0 < n; i0 += XR_U * st) {
        TZ a[XR_U];
        T pi[XR_U], xi[XR_U];
#pragma unroll
        for (int k = 0; k < XR_U; k++) {
            const long i = i0 + k * st;
            if (i >= n) break;
            a[k] = zs[i];
            if (!first) { pi[k] = p[i]; xi[k] = x[i]; }
        }
#pragma unroll
        for (int k = 0; k < XR_U; k++) {
            const long i = i0 + k * st;
            if (i >= n) break;
            const T z = (T)((double)a[k] * sc);
            if (first) {
                p[i] = z;
            } else {
                x[i] = xi[k] + alpha * pi[k];
                p[i] = z + beta * pi[k];
            }
        }
    }
}

// end of an iteration, by one thread: it += 1, rz_prev = rz; optionally set the WHILE condition of the graph
__device__ __forceinline__ void pcg_end(double* scal, cudaGraphConditionalHandle cond, int use_cond) {
    const double it = scal[24] + 1.0;
    scal[24] = it;
    scal[12] = scal[10];
    // learned-correction fallback: off for the rest of the solve once an iteration's residual
    // norm did not drop below ratio x the previous one
    if (scal[28] != 0.0 && scal[29] > 0.0 && !(scal[21] <= scal[27] * scal[27] * scal[29])) scal[28] = 0.0;
    scal[29] = scal[21];
    // precision fallback: the loop ends once |r| has not halved within scal[93] iterations (0: off);
    // scal[90] is the last halving's r.r, scal[91] its iteration, scal[92] the flag
    bool stalled = false;
    if (scal[93] > 0.0) {
        if (scal[21] <= 0.25 * scal[90]) {
            scal[90] = scal[21];
            scal[91] = it;
        } else if (it - scal[91] >= scal[93]) {
            scal[92] = 1.0;
            stalled = true;
        }
    }
    if (use_cond) {
        const double rr = scal[21], bb = scal[22] > 0 ? scal[22] : 1.0;
        const bool go = isfinite(rr) && sqrt(rr) > scal[25] * sqrt(bb) && it < scal[26] && !stalled;
        cudaGraphSetConditional(cond, go ? 1u : 0u);
    }
}

// r -= alpha q, r.r and the end of the iteration (by the last block, which has the sum).  r32 (optional): the new
// residual scaled by 1 / sqrt(rr_old) and rounded to FP32, the right-hand side of the next FP32 V-cycle; rr_old (the r.r
// before this update) is kept in scale_out
template <typename T>
__global__ void __launch_bounds__(RB) k_pcg_r_rr(long n, const double* __restrict__ num, const double* __restrict__ den,
                                                 T* __restrict__ r, const T* __restrict__ q, float* __restrict__ r32,
                                                 const double* rr_old, double* __restrict__ scale_out, RedOut ro,
                                                 double* scal, cudaGraphConditionalHandle cond, int use_cond) {
    const T alpha = den[0] != 0.0 ? (T)(num[0] / den[0]) : T(0);
    const double old = r32 ? rr_old[0] : 0.0, inv = r32 ? 1.0 / sqrt(fmax(old, 1e-300)) : 0.0;
    if (r32 && blockIdx.x == 0 && threadIdx.x == 0) scale_out[0] = old;
    double v[1] = {0};
    // the reduction grid is small (2 blocks per SM): XR_U grid strides per trip keep enough loads in flight
    const long st = (long)gridDim.x * blockDim.x;
    for (long i0 = blockIdx.x * (long)blockDim.x + threadIdx.x; i0 < n; i0 += XR_U * st) {
        T ri[XR_U], qi[XR_U];
#pragma unroll
        for (int k = 0; k < XR_U; k++) {
            const long i = i0 + k * st;
            if (i < n) { ri[k] = r[i]; qi[k] = q[i]; }
        }
#pragma unroll
        for (int k = 0; k < XR_U; k++) {
            const long i = i0 + k * st;
            if (i >= n) break;
            const T rn = ri[k] - alpha * qi[k];
            r[i] = rn;
            if (r32) r32[i] = (float)((double)rn * inv);
            v[0] += (double)rn * (double)rn;
        }
    }
    if (grid_reduce<1>(v, ro) && threadIdx.x == 0) pcg_end(scal, cond, use_cond);
}

// after the loop: the last iteration's step of x (none if the loop did not run)
__global__ void k_pcg_x_last(long n, const double* __restrict__ scal, const double* __restrict__ p, double* __restrict__ x) {
    if (scal[24] == 0.0 || scal[20] == 0.0) return;
    const double alpha = scal[12] / scal[20];
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) x[i] += alpha * p[i];
}

// ---- FP32 Krylov vectors (FP64 accumulation of every dot product) ----------------------
__global__ void __launch_bounds__(RB) k_dot32(long n, const float* __restrict__ a, const float* __restrict__ b,
                                              RedOut ro) {
    double v[1] = {0};
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x)
        v[0] += (double)a[i] * (double)b[i];
    grid_reduce<1>(v, ro);
}

// x += sqrt(s) (d + alpha p): the FP32 correction of a refinement step with its last iteration's step, scaled back to
// the FP64 residual
__global__ void k_axpy_f32_scaled(long n, double* __restrict__ x, const float* __restrict__ d,
                                  const double* __restrict__ s, const double* __restrict__ scal,
                                  const float* __restrict__ p) {
    const double sc = sqrt(fmax(s[0], 0.0));
    const bool step = scal[24] != 0.0 && scal[20] != 0.0;
    const float alpha = step ? (float)(scal[12] / scal[20]) : 0.f;
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x)
        x[i] += sc * (double)(step ? d[i] + alpha * p[i] : d[i]);
}

__global__ void k_scale(long n, double* __restrict__ x, const double* __restrict__ s, int inv_sqrt) {
    const double sc = inv_sqrt ? 1.0 / sqrt(s[0]) : s[0];
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) x[i] *= sc;
}

__device__ __forceinline__ uint64_t splitmix64(uint64_t x) {
    x += 0x9E3779B97F4A7C15ull;
    x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
    x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
    return x ^ (x >> 31);
}
__global__ void k_rng(uint64_t seed, long n, double* __restrict__ out) {
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
        uint64_t hsh = splitmix64(seed * 0x632BE59BD9B4E019ull + (uint64_t)i);
        out[i] = (double)(hsh >> 11) * (1.0 / 9007199254740992.0) * 2.0 - 1.0;
    }
}

// gather load-node values into an AoS [3*nload] vector; optionally keep only the normal component
__global__ void k_gather_load(int nload, long nv, const int* __restrict__ nodes, const double* __restrict__ f,
                              const double* __restrict__ normal, int constrain, double* __restrict__ fs) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nload; i += gridDim.x * blockDim.x) {
        const long v = nodes[i];
        double a = f[v], b = f[nv + v], c = f[2 * nv + v];
        if (constrain) {
            const double n0 = normal[3 * i], n1 = normal[3 * i + 1], n2 = normal[3 * i + 2];
            const double d = a * n0 + b * n1 + c * n2;
            a = d * n0; b = d * n1; c = d * n2;
        }
        fs[3 * i] = a; fs[3 * i + 1] = b; fs[3 * i + 2] = c;
    }
}
__global__ void k_scatter_load(int nload, long nv, const int* __restrict__ nodes, const double* __restrict__ fs,
                               double* __restrict__ f) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nload; i += gridDim.x * blockDim.x) {
        const long v = nodes[i];
        f[v] = fs[3 * i]; f[nv + v] = fs[3 * i + 1]; f[2 * nv + v] = fs[3 * i + 2];
    }
}
// fs -= sum_k (Rd_k . fs) Rd_k with the dots precomputed in w[0..nrig)
__global__ void k_sub_modes(long n, int nrig, const double* __restrict__ Rd, const double* __restrict__ w,
                            double* __restrict__ fs) {
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
        double s = fs[i];
        for (int k = 0; k < nrig; k++) s -= w[k] * Rd[k * n + i];
        fs[i] = s;
    }
}
// six dots against the rigid modes in one pass
__global__ void __launch_bounds__(RB) k_dot6(long n, int nrig, const double* __restrict__ Rd,
                                             const double* __restrict__ x, RedOut ro) {
    double v[6] = {0, 0, 0, 0, 0, 0};
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
        const double xi = x[i];
#pragma unroll
        for (int k = 0; k < 6; k++)
            if (k < nrig) v[k] += Rd[k * n + i] * xi;
    }
    grid_reduce<6>(v, ro);
}

// largest eigenvalue of the symmetric tridiagonal (alpha, beta) by Sturm counts, one warp: each round the 32 lanes
// count at 32 points of the bracket, which shrinks 33-fold, until it is two neighbouring numbers.  One thread's
// bisection took 142 us of dependent divisions, 39 us here (both with the launch).
__global__ void k_tridiag_max(int k, const double* __restrict__ alpha, const double* __restrict__ beta,
                              double* __restrict__ out) {
    const int lane = threadIdx.x & 31;
    double lo = alpha[0], hi = alpha[0];
    for (int i = 0; i < k; i++) {
        const double r = (i > 0 ? fabs(beta[i - 1]) : 0) + (i < k - 1 ? fabs(beta[i]) : 0);
        lo = fmin(lo, alpha[i] - r);
        hi = fmax(hi, alpha[i] + r);
    }
    for (int it = 0; it < 60; it++) {
        const double mid = lo + (hi - lo) * ((lane + 1) / 33.0);
        const bool in = mid > lo && mid < hi;
        bool above = true;  // all k eigenvalues lie below mid
        if (in) {
            int cnt = 0;
            double d = 1;
            for (int i = 0; i < k; i++) {
                const double b2 = i > 0 ? beta[i - 1] * beta[i - 1] : 0;
                d = alpha[i] - mid - (i > 0 ? b2 / d : 0);
                if (d == 0) d = -1e-300;
                if (d < 0) cnt++;
            }
            above = cnt == k;
        }
        const unsigned ins = __ballot_sync(0xffffffffu, in);
        if (ins == 0) break;
        // the points rise with the lane: hi = the first point above the spectrum, lo = the point before it
        const unsigned ab = __ballot_sync(0xffffffffu, in && above), be = __ballot_sync(0xffffffffu, in && !above);
        const double nh = __shfl_sync(0xffffffffu, mid, ab ? __ffs(ab) - 1 : 0);
        const unsigned bl = ab ? be & ((1u << (__ffs(ab) - 1)) - 1u) : be;
        const double nl = __shfl_sync(0xffffffffu, mid, bl ? 31 - __clz(bl) : 0);
        if (ab) hi = nh;
        if (bl) lo = nl;
    }
    if (lane == 0) out[0] = 0.5 * (lo + hi);
}

// the same filter through shared memory, radius (rounded) RL <= 3: a block of 32 x 8 columns keeps the sensitivities
// (0 outside the solid) and the activity of its 32 x 8 x 8 elements and their halo, and the list of taps inside the
// radius with their weights; a thread does 8 elements of a column, so that a tap's entry is read once for them.  Taps
// in k_filter's order, products in FP32 and their sum in FP64 as there.  255x256x128, radius 2:
// 1050 us with 33 bounds-checked gathers per element, 200 us here.
constexpr int FT_Z = 8;
template <int RL>
__global__ void __launch_bounds__(256) k_filter_tile(int nx, int ny, int nz, const uint8_t* __restrict__ eact,
                                                     float radius, const float* __restrict__ sens,
                                                     float* __restrict__ out) {
    constexpr int HX = 32 + 2 * RL, HY = 8 + 2 * RL, HZ = FT_Z + 2 * RL, D = 2 * RL + 1;
    __shared__ float sg[HX * HY * HZ];
    __shared__ uint8_t sa[HX * HY * HZ];
    __shared__ float tw[D * D * D];
    __shared__ int to[D * D * D];
    __shared__ int ntap;
    const int tid = threadIdx.x, x0 = blockIdx.x * 32, y0 = blockIdx.y * 8, z0 = blockIdx.z * FT_Z;
    for (int i = tid; i < HX * HY * HZ; i += 256) {
        const int X = x0 - RL + i % HX, Y = y0 - RL + i / HX % HY, Z = z0 - RL + i / (HX * HY);
        float g = 0.f;
        uint8_t a = 0;
        if (X >= 0 && Y >= 0 && Z >= 0 && X < nx && Y < ny && Z < nz) {
            const long n = X + (long)nx * (Y + (long)ny * Z);
            a = eact[n];
            if (a) g = sens[n];
        }
        sg[i] = g;
        sa[i] = a;
    }
    if (tid == 0) {
        const float R2 = radius * radius;
        int m = 0;
        for (int dx = -RL; dx <= RL; dx++)
            for (int dy = -RL; dy <= RL; dy++)
                for (int dz = -RL; dz <= RL; dz++) {
                    const float r2 = (float)(dx * dx + dy * dy + dz * dz);
                    if (r2 > R2) continue;
                    const float t = sqrtf(r2 / R2);
                    const float t2 = t * t;
                    tw[m] = 1 - 6 * t2 + 8 * t2 * t - 3 * t2 * t2;
                    to[m++] = dx + HX * (dy + HY * dz);
                }
        ntap = m;
    }
    __syncthreads();
    const int lx = tid & 31, ly = tid >> 5, x = x0 + lx, y = y0 + ly;
    if (x >= nx || y >= ny) return;
    const int c = lx + RL + HX * (ly + RL + HY * RL), nt = ntap;
    double gsum[FT_Z];
    float wsum[FT_Z];
#pragma unroll
    for (int k = 0; k < FT_Z; k++) {
        gsum[k] = 0;
        wsum[k] = 0.f;
    }
    for (int i = 0; i < nt; i++) {
        const int o = c + to[i];
        const float wv = tw[i];
#pragma unroll
        for (int k = 0; k < FT_Z; k++)
            if (sa[o + k * HX * HY]) {
                gsum[k] += wv * sg[o + k * HX * HY];
                wsum[k] += wv;
            }
    }
#pragma unroll
    for (int k = 0; k < FT_Z; k++)
        if (z0 + k < nz)
            out[x + (long)nx * (y + (long)ny * (z0 + k))] = sa[c + k * HX * HY] ? (float)(gsum[k] / wsum[k]) : 0.f;
}

// normalised radial sensitivity filter, one thread per element (radii past k_filter_tile's)
__global__ void k_filter(int nx, int ny, int nz, const uint8_t* __restrict__ eact, float radius,
                         const float* __restrict__ sens, float* __restrict__ out) {
    const long ne = (long)nx * ny * nz;
    const float R2 = radius * radius;
    const int Rl = (int)(radius + 0.5f);
    for (long e = blockIdx.x * (long)blockDim.x + threadIdx.x; e < ne; e += (long)gridDim.x * blockDim.x) {
        if (!eact[e]) { out[e] = 0.f; continue; }
        const int x = (int)(e % nx), y = (int)((e / nx) % ny), z = (int)(e / ((long)nx * ny));
        float wsum = 0;
        double gsum = 0;
        for (int dx = -Rl; dx <= Rl; dx++) {
            const int X = x + dx;
            if (X < 0 || X >= nx) continue;
            for (int dy = -Rl; dy <= Rl; dy++) {
                const int Y = y + dy;
                if (Y < 0 || Y >= ny) continue;
                for (int dz = -Rl; dz <= Rl; dz++) {
                    const int Z = z + dz;
                    if (Z < 0 || Z >= nz) continue;
                    const float r2 = (float)(dx * dx + dy * dy + dz * dz);
                    if (r2 > R2) continue;
                    const long n = X + (long)nx * (Y + (long)ny * Z);
                    if (!eact[n]) continue;
                    const float t = sqrtf(r2 / R2);
                    const float t2 = t * t;
                    const float wv = 1 - 6 * t2 + 8 * t2 * t - 3 * t2 * t2;
                    gsum += wv * sens[n];
                    wsum += wv;
                }
            }
        }
        out[e] = (float)(gsum / wsum);
    }
}

__device__ __forceinline__ float clampf(float v, float lo, float hi) { return v < lo ? lo : (v > hi ? hi : v); }

// an element's OC density for the multiplier thr (updateDensities, optimization/optimization.cu:136-162); the default
// damping 1/2 takes the square root instead of a general power
__device__ __forceinline__ float oc_density(float g, float ro, float thr, float step, float damp, float rhomin) {
    if (g > 0) g = 0;
    g = fabsf(g) / thr;
    const float rn = ro * (damp == 0.5f ? sqrtf(g) : powf(g, damp));
    return clampf(clampf(rn, ro - step, ro + step), rhomin, 1.f);
}

// The whole OC update in one cooperative launch: the largest |g|, the bisection of the multiplier on the volume
// (optimization/optimization.cu:164-226) and the update of rho.  The trials read the design from L2 (9 bytes per
// element) and store nothing; the blocks meet at a grid barrier per trial, where every block adds all partial sums in
// the same order and takes the same decision.  res[0] = multiplier, res[1] = trials.  255x256x128: 11 launches of
// 122 us, each followed by a host read-back, before; 25 us per trial here.
__global__ void __launch_bounds__(RB) k_oc_update(long ne, const uint8_t* __restrict__ eact,
                                                  const uint8_t* __restrict__ eshell, float* rho,
                                                  const float* __restrict__ sens, float vgoal, double nact, float step,
                                                  float damp, float rhomin, double* partials, double* __restrict__ res) {
    cg::grid_group grid = cg::this_grid();
    __shared__ double sh[RB / 32];
    const long n4 = ne / 4, st = (long)gridDim.x * RB;
    const long i0 = blockIdx.x * (long)RB + threadIdx.x;
    const uchar4* a4 = reinterpret_cast<const uchar4*>(eact);
    const uchar4* s4 = reinterpret_cast<const uchar4*>(eshell);
    const float4 *r4 = reinterpret_cast<const float4*>(rho), *g4 = reinterpret_cast<const float4*>(sens);
    auto block_sum = [&](double x) {  // the block's sum, in every thread
        __syncthreads();
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
        if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = x;
        __syncthreads();
        double s = 0;
#pragma unroll
        for (int i = 0; i < RB / 32; i++) s += sh[i];
        return s;
    };
    auto block_max = [&](double x) {
        __syncthreads();
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) x = fmax(x, __shfl_xor_sync(0xffffffffu, x, o));
        if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = x;
        __syncthreads();
        double s = 0;
#pragma unroll
        for (int i = 0; i < RB / 32; i++) s = fmax(s, sh[i]);
        return s;
    };
    double m = 0;
    for (long i = i0; i < n4; i += st) {
        const uchar4 a = a4[i];
        const float4 g = g4[i];
        if (a.x) m = fmax(m, (double)fabsf(g.x));
        if (a.y) m = fmax(m, (double)fabsf(g.y));
        if (a.z) m = fmax(m, (double)fabsf(g.z));
        if (a.w) m = fmax(m, (double)fabsf(g.w));
    }
    for (long e = 4 * n4 + i0; e < ne; e += st)
        if (eact[e]) m = fmax(m, (double)fabsf(sens[e]));
    m = block_max(m);
    if (threadIdx.x == 0) partials[blockIdx.x] = m;
    grid.sync();
    double gm = 0;
    for (int i = threadIdx.x; i < (int)gridDim.x; i += RB) gm = fmax(gm, partials[i]);
    gm = block_max(gm);
    auto one = [&](uint8_t a, uint8_t s, float g, float ro, float thr) {
        return !a ? 0.f : s ? 1.f : oc_density(g, ro, thr, step, damp, rhomin);
    };
    float lo = 0, hi = (float)gm, thr = (lo + hi) / 2, V = 2;
    int itn = 0, trials = 0;
    do {
        thr = (lo + hi) / 2;
        double v = 0;
        long i = i0;
        for (; i + st < n4; i += 2 * st) {  // two strides in flight
            const uchar4 a = a4[i], b = a4[i + st], z = make_uchar4(0, 0, 0, 0);
            const uchar4 sa = s4 ? s4[i] : z, sb = s4 ? s4[i + st] : z;
            const float4 g = g4[i], h = g4[i + st], r = r4[i], q = r4[i + st];
            v += ((double)one(a.x, sa.x, g.x, r.x, thr) + (double)one(a.y, sa.y, g.y, r.y, thr)) +
                 ((double)one(a.z, sa.z, g.z, r.z, thr) + (double)one(a.w, sa.w, g.w, r.w, thr));
            v += ((double)one(b.x, sb.x, h.x, q.x, thr) + (double)one(b.y, sb.y, h.y, q.y, thr)) +
                 ((double)one(b.z, sb.z, h.z, q.z, thr) + (double)one(b.w, sb.w, h.w, q.w, thr));
        }
        for (long e = 4 * i; i < n4 && e < 4 * i + 4; e++) v += (double)one(eact[e], eshell ? eshell[e] : 0, sens[e], rho[e], thr);
        for (long e = 4 * n4 + i0; e < ne; e += st) v += (double)one(eact[e], eshell ? eshell[e] : 0, sens[e], rho[e], thr);
        v = block_sum(v);
        // two sets of partial sums by turns: a block may be a trial ahead of another's reads
        double* ps = partials + gridDim.x * (1 + (trials & 1));
        if (threadIdx.x == 0) ps[blockIdx.x] = v;
        grid.sync();
        double vs = 0;
        for (int b = threadIdx.x; b < (int)gridDim.x; b += RB) vs += ps[b];
        vs = block_sum(vs);
        V = (float)(vs / nact);
        trials++;
        if (V > vgoal) lo = thr;
        else if (V < vgoal) hi = thr;
    } while (fabsf(V - vgoal) > 1e-4f && itn++ < 30);
    for (long e = i0; e < ne; e += st) rho[e] = one(eact[e], eshell ? eshell[e] : 0, sens[e], rho[e], thr);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        res[0] = (double)thr;
        res[1] = (double)trials;
    }
}

__global__ void __launch_bounds__(RB) k_count_u8(long n, const uint8_t* __restrict__ a, RedOut ro) {
    double v[1] = {0};
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) v[0] += a[i] ? 1.0 : 0.0;
    grid_reduce<1>(v, ro);
}

__global__ void k_node_active(int nx, int ny, int nz, const uint8_t* __restrict__ eact, uint8_t* __restrict__ vact) {
    const int vx = nx + 1, vy = ny + 1;
    const long nv = (long)vx * vy * (nz + 1);
    for (long v = blockIdx.x * (long)blockDim.x + threadIdx.x; v < nv; v += (long)gridDim.x * blockDim.x) {
        const int x = (int)(v % vx), y = (int)((v / vx) % vy), z = (int)(v / ((long)vx * vy));
        uint8_t a = 0;
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const int ex = x + (i & 1) - 1, ey = y + ((i >> 1) & 1) - 1, ez = z + (i >> 2) - 1;
            if (ex < 0 || ey < 0 || ez < 0 || ex >= nx || ey >= ny || ez >= nz) continue;
            a |= eact[ex + (long)nx * (ey + (long)ny * ez)];
        }
        vact[v] = a ? 1 : 0;
    }
}

__global__ void k_coarsen(int nx, int ny, int nz, int ratio, const uint8_t* __restrict__ ef, uint8_t* __restrict__ ec) {
    const int cx = (nx + ratio - 1) / ratio, cy = (ny + ratio - 1) / ratio, cz = (nz + ratio - 1) / ratio;
    const long nc = (long)cx * cy * cz;
    for (long c = blockIdx.x * (long)blockDim.x + threadIdx.x; c < nc; c += (long)gridDim.x * blockDim.x) {
        const int X = (int)(c % cx), Y = (int)((c / cx) % cy), Z = (int)(c / ((long)cx * cy));
        uint8_t a = 0;
        for (int k = 0; k < ratio && !a; k++)
            for (int j = 0; j < ratio && !a; j++)
                for (int i = 0; i < ratio && !a; i++) {
                    const int x = X * ratio + i, y = Y * ratio + j, z = Z * ratio + k;
                    if (x < nx && y < ny && z < nz) a |= ef[x + (long)nx * (y + (long)ny * z)];
                }
        ec[c] = a ? 1 : 0;
    }
}

__global__ void k_surface(int nx, int ny, int nz, const uint8_t* __restrict__ eact, uint8_t* __restrict__ surf) {
    const int vx = nx + 1, vy = ny + 1;
    const long nv = (long)vx * vy * (nz + 1);
    for (long v = blockIdx.x * (long)blockDim.x + threadIdx.x; v < nv; v += (long)gridDim.x * blockDim.x) {
        const int x = (int)(v % vx), y = (int)((v / vx) % vy), z = (int)(v / ((long)vx * vy));
        bool s[8];
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const int ex = x + (i & 1) - 1, ey = y + ((i >> 1) & 1) - 1, ez = z + (i >> 2) - 1;
            s[i] = (ex >= 0 && ey >= 0 && ez >= 0 && ex < nx && ey < ny && ez < nz) &&
                   eact[ex + (long)nx * (ey + (long)ny * ez)];
        }
        bool ax = false, ay = false, az = false;
#pragma unroll
        for (int i = 0; i < 2; i++)
#pragma unroll
            for (int j = 0; j < 2; j++) {
                // s index = a + 2b + 4c for element offsets (a, b, c) in {0,1}
                ax |= s[0 + 2 * i + 4 * j] && s[1 + 2 * i + 4 * j];
                ay |= s[i + 0 + 4 * j] && s[i + 2 + 4 * j];
                az |= s[i + 2 * j + 0] && s[i + 2 * j + 4];
            }
        surf[v] = (!ax || !ay || !az) ? 1 : 0;
    }
}

__device__ __forceinline__ bool rbit(const uint32_t* b, long id) { return (b[id >> 5] >> (id & 31)) & 1u; }

// one thread per 32-vertex word: no atomics needed
__global__ void k_cube_vbits(int R, const uint32_t* __restrict__ eb, uint32_t* __restrict__ vb) {
    const int V = R + 1;
    const long nvb = (long)V * V * V;
    const long nw = (nvb + 31) / 32;
    for (long wd = blockIdx.x * (long)blockDim.x + threadIdx.x; wd < nw; wd += (long)gridDim.x * blockDim.x) {
        uint32_t word = 0;
        for (int b = 0; b < 32; b++) {
            const long t = wd * 32 + b;
            if (t >= nvb) break;
            const int x = (int)(t % V), y = (int)((t / V) % V), z = (int)(t / ((long)V * V));
            bool a = false;
            for (int i = 0; i < 8 && !a; i++) {
                const int ex = x + (i & 1) - 1, ey = y + ((i >> 1) & 1) - 1, ez = z + (i >> 2) - 1;
                if (ex < 0 || ey < 0 || ez < 0 || ex >= R || ey >= R || ez >= R) continue;
                a = rbit(eb, ex + (long)R * (ey + (long)R * ez));
            }
            if (a) word |= 1u << b;
        }
        vb[wd] = word;
    }
}

__global__ void k_cube_coarsen(int Rf, const uint32_t* __restrict__ ef, uint32_t* __restrict__ ec) {
    const int Rc = Rf >> 1;
    const long nc = (long)Rc * Rc * Rc;
    const long nw = (nc + 31) / 32;
    for (long wd = blockIdx.x * (long)blockDim.x + threadIdx.x; wd < nw; wd += (long)gridDim.x * blockDim.x) {
        uint32_t word = 0;
        for (int b = 0; b < 32; b++) {
            const long t = wd * 32 + b;
            if (t >= nc) break;
            const int X = (int)(t % Rc), Y = (int)((t / Rc) % Rc), Z = (int)(t / ((long)Rc * Rc));
            bool a = false;
            for (int i = 0; i < 8 && !a; i++) {
                const int x = 2 * X + (i & 1), y = 2 * Y + ((i >> 1) & 1), z = 2 * Z + (i >> 2);
                a = rbit(ef, x + (long)Rf * (y + (long)Rf * z));
            }
            if (a) word |= 1u << b;
        }
        ec[wd] = word;
    }
}

// raw rigid-body modes over active nodes: 3 translations, 3 rotations (columns of [p]x)
__global__ void k_rigid_raw(int vx, int vy, long nv, const uint8_t* __restrict__ vact, double* __restrict__ Ru) {
    const long n = 3 * nv;
    for (long v = blockIdx.x * (long)blockDim.x + threadIdx.x; v < nv; v += (long)gridDim.x * blockDim.x) {
        const double a = vact[v] ? 1.0 : 0.0;
        const double px = (double)(v % vx), py = (double)((v / vx) % vy), pz = (double)(v / ((long)vx * vy));
        const double ph[3][3] = {{0, -pz, py}, {pz, 0, -px}, {-py, px, 0}};
        for (int t = 0; t < 3; t++)
            for (int c = 0; c < 3; c++) Ru[(long)t * n + c * nv + v] = (t == c) ? a : 0.0;
        for (int k = 0; k < 3; k++)
            for (int c = 0; c < 3; c++) Ru[(long)(3 + k) * n + c * nv + v] = a * ph[c][k];
    }
}

__global__ void k_axpy_dev(long n, const double* __restrict__ coef, double sign, const double* __restrict__ x,
                           double* __restrict__ y) {
    const double a = sign * coef[0];
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) y[i] += a * x[i];
}

__global__ void k_mask_copy(long n, long nv, const uint8_t* __restrict__ vact, const double* __restrict__ src,
                            double* __restrict__ dst) {
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x)
        dst[i] = vact[i % nv] ? src[i] : 0.0;
}

}  // namespace

namespace rtk {

// the hierarchy's reduction buffers (its launches are ordered on one stream)
static RedOut red(rt_hier* h, double* out) {
    return RedOut{h->partials, out, reinterpret_cast<unsigned*>(h->scal + RT_SCAL_TICKET)};
}

int dot(rt_hier* h, long n, const double* a, const double* b, double* out) {
    return rt_launch(h->ctx, "dot", [&] { k_dot<<<red_grid(n), RB, 0, h->ctx->stream>>>(n, a, b, red(h, out)); });
}

int axpy(rt_hier* h, long n, double a, const double* x, double* y) {
    return rt_launch(h->ctx, "axpy", [&] { k_axpy<<<gridN(h->ctx, n), 256, 0, h->ctx->stream>>>(n, a, x, y); });
}

int f2d(rt_hier* h, long n, const float* a, double* b) {
    return rt_launch(h->ctx, "f2d", [&] { k_f2d<<<gridN(h->ctx, n), 256, 0, h->ctx->stream>>>(n, a, b); });
}

int d2f_scaled(rt_hier* h, long n, const double* a, float* b, const double* s) {
    return rt_launch(h->ctx, "d2f_scaled", [&] { k_d2f_scaled<<<gridN(h->ctx, n), 256, 0, h->ctx->stream>>>(n, a, b, s); });
}

int f2d_scaled(rt_hier* h, long n, const float* a, double* b, const double* s) {
    return rt_launch(h->ctx, "f2d_scaled", [&] { k_f2d_scaled<<<gridN(h->ctx, n), 256, 0, h->ctx->stream>>>(n, a, b, s); });
}

int f2d_scaled_add(rt_hier* h, long n, const float* a, double* b, const double* s) {
    return rt_launch(h->ctx, "f2d_scaled_add",
                     [&] { k_f2d_scaled_add<<<gridN(h->ctx, n), 256, 0, h->ctx->stream>>>(n, a, b, s); });
}

int pcg_zdots(rt_hier* h, long n, const float* z, const double* s, const double* r, const double* q, double* out) {
    return rt_launch(h->ctx, "pcg_zdots", [&] {
        k_pcg_zdots<float, double><<<red_grid(n), RB, 0, h->ctx->stream>>>(n, z, s, r, q, red(h, out));
    });
}
int pcg_zdots(rt_hier* h, long n, const double* z, const double* r, const double* q, double* out) {
    return rt_launch(h->ctx, "pcg_zdots", [&] {
        k_pcg_zdots<double, double><<<red_grid(n), RB, 0, h->ctx->stream>>>(n, z, nullptr, r, q, red(h, out));
    });
}
int pcg_zdots32(rt_hier* h, long n, const float* z, const float* r, const float* q, double* out) {
    return rt_launch(h->ctx, "pcg32_zdots", [&] {
        k_pcg_zdots<float, float><<<red_grid(n), RB, 0, h->ctx->stream>>>(n, z, nullptr, r, q, red(h, out));
    });
}

int pcg_update_xp(rt_hier* h, long n, const float* z, const double* s, double* p, double* x) {
    return rt_launch(h->ctx, "pcg_update_xp", [&] {
        k_pcg_xp<float, double><<<gridN(h->ctx, n), RB, 0, h->ctx->stream>>>(n, h->scal, z, s, p, x);
    });
}
int pcg_update_xp(rt_hier* h, long n, const double* z, double* p, double* x) {
    return rt_launch(h->ctx, "pcg_update_xp", [&] {
        k_pcg_xp<double, double><<<gridN(h->ctx, n), RB, 0, h->ctx->stream>>>(n, h->scal, z, nullptr, p, x);
    });
}
int pcg32_update_xp(rt_hier* h, long n, const float* z, float* p, float* d) {
    return rt_launch(h->ctx, "pcg32_update_xp", [&] {
        k_pcg_xp<float, float><<<gridN(h->ctx, n), RB, 0, h->ctx->stream>>>(n, h->scal, z, nullptr, p, d);
    });
}

int pcg_update_r_rr(rt_hier* h, long n, double* r, const double* q, float* r32, cudaGraphConditionalHandle cond,
                    int use_cond) {
    return rt_launch(h->ctx, "pcg_update_r", [&] {
        k_pcg_r_rr<double><<<red_grid(n), RB, 0, h->ctx->stream>>>(n, h->scal + 10, h->scal + 20, r, q, r32, h->scal + 21,
                                                                   h->scal + 23, red(h, h->scal + 21), h->scal, cond, use_cond);
    });
}
int pcg32_update_r_rr(rt_hier* h, long n, float* r, const float* q, cudaGraphConditionalHandle cond, int use_cond) {
    return rt_launch(h->ctx, "pcg32_update_r", [&] {
        k_pcg_r_rr<float><<<red_grid(n), RB, 0, h->ctx->stream>>>(n, h->scal + 10, h->scal + 20, r, q, nullptr, nullptr,
                                                                  nullptr, red(h, h->scal + 21), h->scal, cond, use_cond);
    });
}

int pcg_x_last(rt_hier* h, long n, double* x) {
    return rt_launch(h->ctx, "pcg_x_last", [&] {
        k_pcg_x_last<<<gridN(h->ctx, n), RB, 0, h->ctx->stream>>>(n, h->scal, h->p, x);
    });
}

int dot32(rt_hier* h, long n, const float* a, const float* b, double* out) {
    return rt_launch(h->ctx, "dot32", [&] { k_dot32<<<red_grid(n), RB, 0, h->ctx->stream>>>(n, a, b, red(h, out)); });
}

int axpy_f32_scaled(rt_hier* h, long n, double* x, const float* d, const double* s) {
    return rt_launch(h->ctx, "axpy_f32", [&] {
        k_axpy_f32_scaled<<<gridN(h->ctx, n), 256, 0, h->ctx->stream>>>(n, x, d, s, h->scal, h->p32k);
    });
}

int scale(rt_hier* h, long n, double* x, const double* s, bool inv_sqrt) {
    return rt_launch(h->ctx, "scale", [&] { k_scale<<<gridN(h->ctx, n), 256, 0, h->ctx->stream>>>(n, x, s, inv_sqrt ? 1 : 0); });
}

int mask_copy(rt_hier* h, long n, const double* src, double* dst) {
    rt_level& L = h->L[0];
    return rt_launch(h->ctx, "mask_copy",
                     [&] { k_mask_copy<<<gridN(h->ctx, n), 256, 0, h->ctx->stream>>>(n, L.nv, L.vact, src, dst); });
}

int rng_uniform(rt_hier* h, uint64_t seed, long n, double* out) {
    return rt_launch(h->ctx, "rng_uniform", [&] { k_rng<<<gridN(h->ctx, n), 256, 0, h->ctx->stream>>>(seed, n, out); });
}

int gather_load(rt_hier* h, const double* f, double* fs) {
    if (h->nload == 0) return RT_OK;
    return rt_launch(h->ctx, "gather_load", [&] {
        k_gather_load<<<gridN(h->ctx, h->nload), 256, 0, h->ctx->stream>>>(h->nload, h->L[0].nv, h->load_nodes, f,
                                                                          h->load_normal, 0, fs);
    });
}

int scatter_load(rt_hier* h, const double* fs, double* f) {
    if (h->nload == 0) return RT_OK;
    return rt_launch(h->ctx, "scatter_load", [&] {
        k_scatter_load<<<gridN(h->ctx, h->nload), 256, 0, h->ctx->stream>>>(h->nload, h->L[0].nv, h->load_nodes, fs, f);
    });
}

// forceProject: gather -> (normal part) -> minus rigid part -> zero f -> scatter
int project_load(rt_hier* h, double* f) {
    rt_level& L = h->L[0];
    const int constrain = (h->P.mode == RT_MODE_NSCF || h->P.mode == RT_MODE_WSCF) ? 1 : 0;
    const long n = 3L * h->nload;
    if (h->nload > 0)
        RT_CHECK(rt_launch(h->ctx, "gather_load", [&] {
            k_gather_load<<<gridN(h->ctx, h->nload), 256, 0, h->ctx->stream>>>(h->nload, L.nv, h->load_nodes, f,
                                                                              h->load_normal, constrain, h->fs);
        }));
    if (h->nrig > 0 && n > 0) {
        RT_CHECK(rt_launch(h->ctx, "dot6", [&] {
            k_dot6<<<red_grid(n), RB, 0, h->ctx->stream>>>(n, h->nrig, h->Rd, h->fs, red(h, h->scal + 40));
        }));
        RT_CHECK(rt_launch(h->ctx, "sub_modes", [&] {
            k_sub_modes<<<gridN(h->ctx, n), 256, 0, h->ctx->stream>>>(n, h->nrig, h->Rd, h->scal + 40, h->fs);
        }));
    }
    RT_CUDA(h->ctx, cudaMemsetAsync(f, 0, sizeof(double) * 3 * L.nv, h->ctx->stream));
    return scatter_load(h, h->fs, f);
}

int displacement_project(rt_hier* h, double* u) {
    rt_level& L = h->L[0];
    const long n = 3 * L.nv;
    RT_CHECK(rt_launch(h->ctx, "dot6", [&] {
        k_dot6<<<red_grid(n), RB, 0, h->ctx->stream>>>(n, 6, h->Ru, u, red(h, h->scal + 40));
    }));
    return rt_launch(h->ctx, "sub_modes",
                     [&] { k_sub_modes<<<gridN(h->ctx, n), 256, 0, h->ctx->stream>>>(n, 6, h->Ru, h->scal + 40, u); });
}

// setNodes (optimization/projection.cpp:46-127): orthonormal rigid modes over all active nodes
int rigid_nodes(rt_hier* h) {
    rt_level& L = h->L[0];
    const long n = 3 * L.nv;
    if (h->Ru == nullptr && cudaMalloc(&h->Ru, sizeof(double) * 6 * n) != cudaSuccess) {
        cudaGetLastError();
        return rt_fail(h->ctx, RT_ENOMEM, "rigid modes: allocation failed");
    }
    RT_CHECK(rt_launch(h->ctx, "rigid_raw", [&] {
        k_rigid_raw<<<gridN(h->ctx, L.nv), 256, 0, h->ctx->stream>>>(L.vx, L.vy, L.nv, L.vact, h->Ru);
    }));
    for (int a = 0; a < 6; a++) {
        double* ra = h->Ru + a * n;
        for (int b = 0; b < a; b++) {
            RT_CHECK(dot(h, n, ra, h->Ru + b * n, h->scal + 70));
            RT_CHECK(rt_launch(h->ctx, "axpy_dev", [&] {
                k_axpy_dev<<<gridN(h->ctx, n), 256, 0, h->ctx->stream>>>(n, h->scal + 70, -1.0, h->Ru + b * n, ra);
            }));
        }
        RT_CHECK(dot(h, n, ra, ra, h->scal + 71));
        RT_CHECK(scale(h, n, ra, h->scal + 71, true));
    }
    return RT_OK;
}

int tridiag_max_eig(rt_hier* h, int k, const double* a, const double* b, double* out) {
    return rt_launch(h->ctx, "tridiag_max", [&] { k_tridiag_max<<<1, 32, 0, h->ctx->stream>>>(k, a, b, out); });
}

int filter(rt_hier* h, float radius) {
    rt_level& L = h->L[0];
    RT_CUDA(h->ctx, cudaMemcpyAsync(h->ftmp, h->sens, sizeof(float) * L.ne, cudaMemcpyDeviceToDevice, h->ctx->stream));
    const dim3 g((L.nx + 31) / 32, (L.ny + 7) / 8, (L.nz + FT_Z - 1) / FT_Z);
    return rt_launch(h->ctx, "filter", [&] {
        const int Rl = (int)(radius + 0.5f);
        if (Rl <= 1)
            k_filter_tile<1><<<g, 256, 0, h->ctx->stream>>>(L.nx, L.ny, L.nz, L.eact, radius, h->ftmp, h->sens);
        else if (Rl == 2)
            k_filter_tile<2><<<g, 256, 0, h->ctx->stream>>>(L.nx, L.ny, L.nz, L.eact, radius, h->ftmp, h->sens);
        else if (Rl == 3)
            k_filter_tile<3><<<g, 256, 0, h->ctx->stream>>>(L.nx, L.ny, L.nz, L.eact, radius, h->ftmp, h->sens);
        else
            k_filter<<<gridN(h->ctx, L.ne), 256, 0, h->ctx->stream>>>(L.nx, L.ny, L.nz, L.eact, radius, h->ftmp, h->sens);
    });
}

int oc_update(rt_hier* h, float vgoal, double* res) {
    rt_level& L = h->L[0];
    rt_ctx* c = h->ctx;
    int nb = 0;
    RT_CUDA(c, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_oc_update, RB, 0));
    if (nb < 1) return rt_fail(c, RT_ECUDA, "cooperative launch unavailable");
    // 3 sets of partials (RT_PARTIALS holds 64 per SM)
    const long want = (L.ne / 4 + RB - 1) / RB, cap = (long)c->sm_count * (nb < 4 ? nb : 4);
    const unsigned g = (unsigned)(want < 1 ? 1 : want < cap ? want : cap);
    long ne = L.ne;
    const uint8_t *ea = L.eact, *es = h->eshell;
    float *rho = h->rho, step = h->P.design_step, damp = h->P.damp_ratio, rmin = h->P.min_rho;
    const float* sens = h->sens;
    double nact = (double)L.n_act_elems, *part = h->partials;
    void* args[] = {&ne, &ea, &es, &rho, &sens, &vgoal, &nact, &step, &damp, &rmin, &part, &res};
    cudaError_t e = cudaSuccess;
    RT_CHECK(rt_launch(c, "oc_update", [&] {
        e = cudaLaunchCooperativeKernel((void*)k_oc_update, g, RB, args, 0, c->stream);
    }));
    if (e != cudaSuccess) return rt_fail(c, RT_ECUDA, "OC update launch failed: %s", cudaGetErrorString(e));
    return RT_OK;
}

int count_u8(rt_ctx* c, long n, const uint8_t* a, double* out) {
    double* part = nullptr;  // partial sums and, after them, the ticket
    RT_CUDA(c, cudaMallocAsync(&part, sizeof(double) * (RT_RED_BLOCKS + 1), c->stream));
    RT_CUDA(c, cudaMemsetAsync(part + RT_RED_BLOCKS, 0, sizeof(double), c->stream));
    RT_CHECK(rt_launch(c, "count_u8", [&] {
        k_count_u8<<<RT_RED_BLOCKS, RB, 0, c->stream>>>(n, a, RedOut{part, out, reinterpret_cast<unsigned*>(part + RT_RED_BLOCKS)});
    }));
    RT_CUDA(c, cudaFreeAsync(part, c->stream));
    return RT_OK;
}

int node_active(rt_ctx* c, int nx, int ny, int nz, const uint8_t* eact, uint8_t* vact) {
    long nv = (long)(nx + 1) * (ny + 1) * (nz + 1);
    return rt_launch(c, "node_active", [&] { k_node_active<<<gridN(c, nv), 256, 0, c->stream>>>(nx, ny, nz, eact, vact); });
}

int coarsen_elements(rt_ctx* c, int nx, int ny, int nz, int ratio, const uint8_t* ef, uint8_t* ec) {
    long nc = (long)((nx + ratio - 1) / ratio) * ((ny + ratio - 1) / ratio) * ((nz + ratio - 1) / ratio);
    return rt_launch(c, "coarsen_elements",
                     [&] { k_coarsen<<<gridN(c, nc), 256, 0, c->stream>>>(nx, ny, nz, ratio, ef, ec); });
}

int surface_nodes(rt_hier* h, uint8_t* surf) {
    rt_level& L = h->L[0];
    return rt_launch(h->ctx, "surface_nodes",
                     [&] { k_surface<<<gridN(h->ctx, L.nv), 256, 0, h->ctx->stream>>>(L.nx, L.ny, L.nz, L.eact, surf); });
}

int cube_vbits(rt_ctx* c, int R, const uint32_t* eb, uint32_t* vb) {
    long nw = ((long)(R + 1) * (R + 1) * (R + 1) + 31) / 32;
    return rt_launch(c, "cube_vbits", [&] { k_cube_vbits<<<gridN(c, nw), 256, 0, c->stream>>>(R, eb, vb); });
}

int cube_coarsen(rt_ctx* c, int R, const uint32_t* ef, uint32_t* ec) {
    long nw = ((long)(R / 2) * (R / 2) * (R / 2) + 31) / 32;
    return rt_launch(c, "cube_coarsen", [&] { k_cube_coarsen<<<gridN(c, nw), 256, 0, c->stream>>>(R, ef, ec); });
}

}  // namespace rtk
