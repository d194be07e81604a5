// rt_coarse.cu — assembled-stencil levels, grid transfers and Galerkin assembly.
//
// Restates:
//   update_residual_kernel_1               grid/Grid.cu:1350-1448
//   gs_relax_kernel                        grid/Grid.cu:678-790
//   restrict_residual{,_nondyadic}_kernel  grid/Grid.cu:1680-1794
//   prolongate_correction{,_nondyadic}_kernel grid/Grid.cu:1818-1895
//   restrict_stencil_nondyadic_OTFA_{NS,WS}_kernel grid/Grid.cu:296-506
//   restrict_stencil_dyadic_kernel         grid/Grid.cu:120-177
// Stencils are [27*9][nv]: entry (k*9 + 3*row + col)*nv + v couples node v to
// neighbour v + d(k), d(k) = (k%3-1, k/3%3-1, k/9-1) — the reference's
// GraftArray<double,27,9> layout over a dense node box.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "rt_internal.h"
#include "rt_tc.cuh"

namespace {

constexpr int ST_BS = 256;

unsigned grid_for(rt_ctx* c, long n, int bs) {
    long b = rt_blocks(n, bs);
    long cap = (long)c->sm_count * 16;
    return (unsigned)(b < cap ? b : cap);
}

// ---------------------------------------------------------------------------
// Stencil storage.  The assembled FP64 operator is row-major, row j = 9 k + 3 r + c
// (neighbour k, block row r, column c) of all nodes: [243][nv].  The FP32 and BF16
// copies the smoothers read are blocked by 32 nodes, [nv/32][RS][32]: the rows of 32
// neighbouring nodes form one contiguous run (31 KB in FP32), so the loads of a warp
// stay in one or two DRAM pages and TLB entries instead of touching 243 rows nv apart.
// The BF16 copy has 9 more rows (RS = 252): the centre block is stored as hi + lo
// BF16 pairs, and is shifted by the rounding error of the 26 off-centre blocks, so
// the row sums of every 3x3 block row (the operator applied to the three rigid
// translations) equal the FP64 operator's to ~2^-17 instead of ~2^-9.
// ---------------------------------------------------------------------------
template <typename S>
struct StAddr {
    static constexpr bool BLK = sizeof(S) < 8;
    static constexpr int RS = sizeof(S) == 2 ? 252 : 243;
    __device__ __forceinline__ static long base(long v) { return BLK ? (v >> 5) * (RS * 32L) + (v & 31) : v; }
    __device__ __forceinline__ static long stride(long nv) { return BLK ? 32 : nv; }
};

// a stencil entry in the compute type: FP64 / FP32 as stored, BF16 bit patterns widened exactly
template <typename T>
__device__ __forceinline__ T st_val(const T* p) { return *p; }
__device__ __forceinline__ float st_val(const uint16_t* p) { return __uint_as_float((uint32_t)*p << 16); }

// entry (block row r, column c) of the centre block; sb = st + StAddr::base(v)
template <typename T, typename S>
__device__ __forceinline__ T st_centre(const S* sb, long rs, int rc) {
    T x = (T)st_val(sb + (117 + rc) * rs);
    if (sizeof(S) == 2) x += (T)st_val(sb + (243 + rc) * rs);
    return x;
}

// one colour of the point-block GS on a stencil level, LPN lanes per node: lane q sums neighbours k = q, q + LPN, ...
// (the low lane bits count nodes, so that neighbouring lanes read neighbouring columns).  A colour of the levels below
// the first has tens to hundreds of nodes, where a thread's 27 x 12 loads one after another took 16 us with the
// launch; 4 lanes where the colour's nodes fill the GPU, a warp per node below that: 8 us.
template <typename T, int LPN>
__global__ void __launch_bounds__(128) k_st_gs(int vx, int vy, int vz, int color, bool backward,
                                               const uint8_t* __restrict__ vact, const T* __restrict__ st,
                                               T* __restrict__ u, const T* __restrict__ f) {
    constexpr int NPW = 32 / LPN;  // nodes per warp
    const long nv = (long)vx * vy * vz;
    const long rs = StAddr<T>::stride(nv);
    const int px = color & 1, py = (color >> 1) & 1, pz = (color >> 2) & 1;
    const int cx = (vx - px + 1) / 2, cy = (vy - py + 1) / 2, cz = (vz - pz + 1) / 2;
    const int nc = cx * cy * cz;
    const int lane = threadIdx.x & 31, q = lane / NPW;
    const int stride = gridDim.x * 4 * NPW;
    for (int t0 = (blockIdx.x * 4 + (threadIdx.x >> 5)) * NPW; t0 < nc; t0 += stride) {
        const int t = t0 + lane % NPW;
        T Au[3] = {T(0), T(0), T(0)}, S[9], F[3], uu[3];
        long v = 0;
        bool act = false;
        if (t < nc) {
            const int x = px + 2 * (t % cx), y = py + 2 * (t / cx % cy), z = pz + 2 * (t / (cx * cy));
            v = x + (long)vx * (y + (long)vy * z);
            act = vact[v];
            const T* sb = st + StAddr<T>::base(v);
            if (act && q == 0) {
#pragma unroll
                for (int i = 0; i < 9; i++) S[i] = st_centre<T>(sb, rs, i);
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    F[c] = f[c * nv + v];
                    uu[c] = u[c * nv + v];
                }
            }
            if (act)
#pragma unroll
                for (int kk = 0; kk < (27 + LPN - 1) / LPN; kk++) {
                    const int k = q + LPN * kk;
                    const int jx = x + k % 3 - 1, jy = y + (k / 3) % 3 - 1, jz = z + k / 9 - 1;
                    if (k >= 27 || k == 13 || jx < 0 || jy < 0 || jz < 0 || jx >= vx || jy >= vy || jz >= vz) continue;
                    const long nj = jx + (long)vx * (jy + (long)vy * jz);
                    const T u0 = u[nj], u1 = u[nv + nj], u2 = u[2 * nv + nj];
#pragma unroll
                    for (int r = 0; r < 3; r++) {
                        const T* s = sb + (long)(k * 9 + 3 * r) * rs;
                        Au[r] += s[0] * u0 + s[rs] * u1 + s[2 * rs] * u2;
                    }
                }
        }
#pragma unroll
        for (int o = NPW; o < 32; o <<= 1)
#pragma unroll
            for (int r = 0; r < 3; r++) Au[r] += __shfl_xor_sync(0xffffffffu, Au[r], o);
        if (!act || q != 0) continue;
        if (!backward) {
            uu[0] = (F[0] - S[1] * uu[1] - S[2] * uu[2] - Au[0]) / S[0];
            uu[1] = (F[1] - S[3] * uu[0] - S[5] * uu[2] - Au[1]) / S[4];
            uu[2] = (F[2] - S[6] * uu[0] - S[7] * uu[1] - Au[2]) / S[8];
        } else {
            uu[2] = (F[2] - S[6] * uu[0] - S[7] * uu[1] - Au[2]) / S[8];
            uu[1] = (F[1] - S[3] * uu[0] - S[5] * uu[2] - Au[1]) / S[4];
            uu[0] = (F[0] - S[1] * uu[1] - S[2] * uu[2] - Au[0]) / S[0];
        }
        u[v] = uu[0]; u[nv + v] = uu[1]; u[2 * nv + v] = uu[2];
    }
}

// ---------------------------------------------------------------------------
// Stencil kernels, a block per 32 nodes: warp j sums the three neighbours k = 3 j .. 3 j + 2 of its lane's node, so
// that every load of a stencil row is a whole line of the blocked layout, and the partial sums meet in shared memory.
// MODE 0: r = f - A u;  MODE 2: Jacobi;  MODE 3: Chebyshev step.
// 4 to 32 lanes per node touched 4 to 16 lines a load.  FP32 Chebyshev, 8 steps in a graph: 882 nodes 29 -> 21 us, 5746
// nodes 43 (4 lanes) -> 23 us; 342k nodes a step 64 us, 5.3 TB/s of stencils, where the bulk-copy form takes 124 us.
// ---------------------------------------------------------------------------
template <typename T, int MODE, typename S>
__global__ void __launch_bounds__(288) k_st_tile(int vx, int vy, int vz, const uint8_t* __restrict__ vact,
                                                 const S* __restrict__ st, const T* __restrict__ u,
                                                 const T* __restrict__ f, T* __restrict__ out, T* __restrict__ d,
                                                 T omega, const double* __restrict__ coef, int kstep) {
    __shared__ T red[9][3][32];
    T ca = T(0), cb = T(0);
    if (MODE == 3) {
        ca = (T)coef[2 * kstep];
        cb = (T)coef[2 * kstep + 1];
    }
    const int nv = vx * vy * vz;  // 243 nv < 2^31
    const long rs = StAddr<S>::stride(nv);
    const int lane = threadIdx.x & 31, j = threadIdx.x >> 5, v = blockIdx.x * 32 + lane;
    const bool inb = v < nv, act = inb && vact[v];
    const S* sb = st + StAddr<S>::base(inb ? v : 0);
    const int oq = j * nv + v;  // warp j (0..2) owns component j
    T S9[9], f0 = T(0), f1 = T(0), f2 = T(0), uo = T(0), dl = T(0);
    if (j < 3 && inb) {
        if (MODE == 0) {
            f0 = f[oq];
        } else {
#pragma unroll
            for (int i = 0; i < 9; i++) S9[i] = st_centre<T>(sb, rs, i);
            f0 = f[v];
            f1 = f[nv + v];
            f2 = f[2 * nv + v];
            uo = u[oq];
            if (MODE == 3 && kstep > 0) dl = d[oq];
        }
    }
    T Au[3] = {T(0), T(0), T(0)};
    const int x = v % vx, y = v / vx % vy, z = v / (vx * vy), jy = y + j % 3 - 1, jz = z + j / 3 - 1;
    if (act && jy >= 0 && jz >= 0 && jy < vy && jz < vz) {
        const int n0 = x + vx * (jy + vy * jz);
        T un[3][3];  // outside the box zero; the stencil has entries there too
#pragma unroll
        for (int i = 0; i < 3; i++)
#pragma unroll
            for (int c = 0; c < 3; c++) un[i][c] = x + i - 1 >= 0 && x + i - 1 < vx ? u[c * nv + n0 + i - 1] : T(0);
#pragma unroll
        for (int i = 0; i < 3; i++) {
            const int k = 3 * j + i;
            const S* s = sb + (long)(k * 9) * rs;
#pragma unroll
            for (int r = 0; r < 3; r++) {
                T a[3];
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    a[c] = (T)st_val(s + (3 * r + c) * rs);
                    // low parts of the BF16 centre block
                    if (sizeof(S) == 2 && k == 13) a[c] += (T)st_val(sb + (243 + 3 * r + c) * rs);
                }
                Au[r] += a[0] * un[i][0] + a[1] * un[i][1] + a[2] * un[i][2];
            }
        }
    }
#pragma unroll
    for (int r = 0; r < 3; r++) red[j][r][lane] = Au[r];
    __syncthreads();
    if (j >= 3 || !inb) return;
    if (MODE == 0) {
        T a = T(0);
#pragma unroll
        for (int i = 0; i < 9; i++) a += red[i][j][lane];
        out[oq] = act ? f0 - a : T(0);
        return;
    }
#pragma unroll
    for (int r = 0; r < 3; r++) {
        Au[r] = T(0);
#pragma unroll
        for (int i = 0; i < 9; i++) Au[r] += red[i][r][lane];
    }
    T res = T(0), dn = T(0);
    if (act) {
        const T A = S9[4] * S9[8] - S9[5] * S9[7], B = S9[5] * S9[6] - S9[3] * S9[8], C = S9[3] * S9[7] - S9[4] * S9[6];
        const T id = T(1) / (S9[0] * A + S9[1] * B + S9[2] * C);
        // row j of the inverse (adjugate / determinant)
        const T i0 = j == 0 ? A : j == 1 ? B : C;
        const T i1 = j == 0   ? S9[2] * S9[7] - S9[1] * S9[8]
                     : j == 1 ? S9[0] * S9[8] - S9[2] * S9[6]
                              : S9[1] * S9[6] - S9[0] * S9[7];
        const T i2 = j == 0   ? S9[1] * S9[5] - S9[2] * S9[4]
                     : j == 1 ? S9[2] * S9[3] - S9[0] * S9[5]
                              : S9[0] * S9[4] - S9[1] * S9[3];
        const T zz = id * (i0 * (f0 - Au[0]) + i1 * (f1 - Au[1]) + i2 * (f2 - Au[2]));
        if (MODE == 2) {
            res = uo + omega * zz;
        } else {
            dn = ca * dl + cb * zz;  // dl = 0 in step 0
            res = uo + dn;
        }
    }
    out[oq] = res;
    if (MODE == 3) d[oq] = dn;
}

// one smoothing step from u = 0: out = omega D^-1 f (MODE 2) or out = d = b_0 D^-1 f (MODE 3), D the centre block;
// it reads 9 of the 243 stencil rows
template <typename T, int MODE, typename S = T>
__global__ void __launch_bounds__(128) k_st_diag(long nv, const uint8_t* __restrict__ vact, const S* __restrict__ st,
                                                 const T* __restrict__ f, T* __restrict__ out, T* __restrict__ d,
                                                 T omega, const double* __restrict__ coef) {
    const T scale = MODE == 3 ? (T)coef[1] : omega;
    const long rs = StAddr<S>::stride(nv);
    for (long v = blockIdx.x * (long)blockDim.x + threadIdx.x; v < nv; v += (long)gridDim.x * blockDim.x) {
        const bool act = vact[v];
        const S* sb = st + StAddr<S>::base(v);
        T m[9];
#pragma unroll
        for (int i = 0; i < 9; i++) m[i] = st_centre<T>(sb, rs, i);
        const T f0 = f[v], f1 = f[nv + v], f2 = f[2 * nv + v];
        T o[3] = {T(0), T(0), T(0)};
        if (act) {
            const T A = m[4] * m[8] - m[5] * m[7], B = m[5] * m[6] - m[3] * m[8], Cc = m[3] * m[7] - m[4] * m[6];
            const T id = T(1) / (m[0] * A + m[1] * B + m[2] * Cc) * scale;
            o[0] = id * (A * f0 + (m[2] * m[7] - m[1] * m[8]) * f1 + (m[1] * m[5] - m[2] * m[4]) * f2);
            o[1] = id * (B * f0 + (m[0] * m[8] - m[2] * m[6]) * f1 + (m[2] * m[3] - m[0] * m[5]) * f2);
            o[2] = id * (Cc * f0 + (m[1] * m[6] - m[0] * m[7]) * f1 + (m[0] * m[4] - m[1] * m[3]) * f2);
        }
#pragma unroll
        for (int q = 0; q < 3; q++) {
            out[q * nv + v] = o[q];
            if (MODE == 3) d[q * nv + v] = o[q];
        }
    }
}

// ---------------------------------------------------------------------------
// Fused Chebyshev sweeps of a small stencil level: all nsteps steps in one cooperative
// launch, the steps separated by a grid barrier instead of a kernel boundary.  The coarse
// levels below the first are a few thousand nodes: a separate launch per step spends most
// of its time in launch, ramp-up and drain, not in the 243-entry rows.  4 lanes per node, lane q sums
// neighbours k = q, q + 4, ...; u is ping-ponged with tmp (u -> tmp -> u ...), so
// after an odd step count a last barrier lets every thread copy its own entries back to u.
// Values written by other blocks in the previous step are read through L2 (ld.global.cg):
// L1 is not coherent across SMs.  The barrier is bounded: a block whose wait runs out sets
// the error slot, poisons u[0] with NaN (the solve then stops on its NaN check) and returns.
// ---------------------------------------------------------------------------
// the polls of a wait come from the context (rt_ctx_set_wait_limit; default 1 << 22, a few hundred
// ns each at most)

__device__ __forceinline__ unsigned ld_acquire_u32(const unsigned* p) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// grid-wide barrier: bar[0] counts arrivals, bar[1] is the generation; gen is thread 0's copy
__device__ __forceinline__ bool coop_grid_sync(unsigned* bar, unsigned& gen, int* s_ok, long spin_limit) {
    __syncthreads();
    if (threadIdx.x == 0) {
        bool ok = true;
        __threadfence();
        const unsigned prev = atomicAdd(bar, 1u);
        if (prev == gridDim.x - 1) {
            atomicExch(bar, 0u);
            __threadfence();
            atomicExch(bar + 1, gen + 1);
        } else {
            long it = 0;
            while (ld_acquire_u32(bar + 1) == gen) {
                if (++it > spin_limit) {
                    ok = false;
                    break;
                }
            }
        }
        __threadfence();
        gen++;
        *s_ok = ok ? 1 : 0;
    }
    __syncthreads();
    return *s_ok != 0;
}

template <typename S>
__global__ void __launch_bounds__(ST_BS, 3) k_st_cheby_coop(int nx, int ny, int nz, const uint8_t* __restrict__ vact,
                                                             const S* __restrict__ st, float* u,
                                                             const float* __restrict__ f, float* tmp, float* d,
                                                             const double* __restrict__ coef, int nsteps,
                                                             unsigned* bar, double* err, long spin_limit) {
    __shared__ int s_ok;
    unsigned gen = 0;
    if (threadIdx.x == 0) gen = ld_acquire_u32(bar + 1);
    const int vx = nx + 1, vy = ny + 1, vz = nz + 1;
    const long nv = (long)vx * vy * vz;
    const long rs = StAddr<S>::stride(nv);
    const int q = threadIdx.x & 3;
    const long ngroups = (long)gridDim.x * (blockDim.x >> 2);
    const long vend = ((nv + ngroups - 1) / ngroups) * ngroups;
    const long v0 = (blockIdx.x * (long)blockDim.x + threadIdx.x) >> 2;
    for (int s = 0; s < nsteps; s++) {
        const float* src = (s & 1) ? tmp : u;
        float* dst = (s & 1) ? u : tmp;
        const float ca = (float)coef[2 * s], cb = (float)coef[2 * s + 1];
        for (long v = v0; v < vend; v += ngroups) {
            const bool inb = v < nv;
            const bool act = inb && vact[v];
            const S* sb = st + StAddr<S>::base(inb ? v : 0);
            float Au[3] = {0.f, 0.f, 0.f};
            if (act) {
                const int x = (int)(v % vx), y = (int)((v / vx) % vy), z = (int)(v / ((long)vx * vy));
#pragma unroll
                for (int kk = 0; kk < 7; kk++) {
                    const int k = q + 4 * kk;
                    if (k >= 27) break;
                    const int jx = x + k % 3 - 1, jy = y + (k / 3) % 3 - 1, jz = z + k / 9 - 1;
                    if (jx < 0 || jy < 0 || jz < 0 || jx >= vx || jy >= vy || jz >= vz) continue;
                    const long nj = jx + (long)vx * (jy + (long)vy * jz);
                    const float u0 = __ldcg(src + nj), u1 = __ldcg(src + nv + nj), u2 = __ldcg(src + 2 * nv + nj);
                    const S* sk = sb + (long)(k * 9) * rs;
#pragma unroll
                    for (int r = 0; r < 3; r++) {
                        float a0 = st_val(sk + (3 * r) * rs), a1 = st_val(sk + (3 * r + 1) * rs),
                              a2 = st_val(sk + (3 * r + 2) * rs);
                        if (sizeof(S) == 2 && k == 13) {  // low parts of the BF16 centre block
                            a0 += st_val(sb + (243 + 3 * r) * rs);
                            a1 += st_val(sb + (243 + 3 * r + 1) * rs);
                            a2 += st_val(sb + (243 + 3 * r + 2) * rs);
                        }
                        Au[r] += a0 * u0 + a1 * u1 + a2 * u2;
                    }
                }
            }
#pragma unroll
            for (int r = 0; r < 3; r++) {
                Au[r] += __shfl_xor_sync(0xffffffffu, Au[r], 1);
                Au[r] += __shfl_xor_sync(0xffffffffu, Au[r], 2);
            }
            if (!inb || q == 3) continue;
            const long oq = (long)q * nv + v;
            float res = 0.f, dn = 0.f;
            if (act) {
                float S9[9];
#pragma unroll
                for (int i = 0; i < 9; i++) S9[i] = st_centre<float>(sb, rs, i);
                const float a0 = S9[0], b0 = S9[1], c0 = S9[2], d0 = S9[3], e0 = S9[4], f0 = S9[5], g0 = S9[6],
                            h0 = S9[7], k0 = S9[8];
                const float A = e0 * k0 - f0 * h0, B = -(d0 * k0 - f0 * g0), Cc = d0 * h0 - e0 * g0;
                const float id = 1.f / (a0 * A + b0 * B + c0 * Cc);
                const float i0 = q == 0 ? A : (q == 1 ? B : Cc);
                const float i1 = q == 0 ? -(b0 * k0 - c0 * h0) : (q == 1 ? (a0 * k0 - c0 * g0) : -(a0 * h0 - b0 * g0));
                const float i2 = q == 0 ? (b0 * f0 - c0 * e0) : (q == 1 ? -(a0 * f0 - c0 * d0) : (a0 * e0 - b0 * d0));
                const float r0 = f[v] - Au[0], r1 = f[nv + v] - Au[1], r2 = f[2 * nv + v] - Au[2];
                const float zq = (i0 * id) * r0 + (i1 * id) * r1 + (i2 * id) * r2;
                dn = (s == 0 ? 0.f : ca * d[oq]) + cb * zq;
                res = __ldcg(src + oq) + dn;
            }
            dst[oq] = res;
            d[oq] = dn;
        }
        if (s + 1 < nsteps || (nsteps & 1)) {
            if (!coop_grid_sync(bar, gen, &s_ok, spin_limit)) {
                if (threadIdx.x == 0) {
                    *err = 2.0;
                    u[0] = __int_as_float(0x7fc00000);
                }
                return;
            }
        }
    }
    if (nsteps & 1) {  // the last step wrote tmp: every thread copies back the entries it wrote
        for (long v = v0; v < nv; v += ngroups)
            if (q < 3) u[(long)q * nv + v] = __ldcg(tmp + (long)q * nv + v);
    }
}

// Resident form of the fused sweeps, for levels whose 4-lane groups all fit on the device at
// once (one group per node, 64 nodes per block): the stencil rows each lane multiplies are
// read once into shared memory (63 x 256 floats, entries outside the box or of inactive
// nodes zeroed so the step has no bounds branches), the inverse diagonal row, f and the
// Chebyshev direction stay in registers, and a step moves only the neighbours' u through L2.
constexpr int RES_ROWS = 63;  // 7 neighbours x 9 entries per lane
constexpr size_t RES_SMEM = (size_t)RES_ROWS * ST_BS * sizeof(float);

template <typename S>
__global__ void __launch_bounds__(ST_BS, 3) k_st_cheby_res(int nx, int ny, int nz, const uint8_t* __restrict__ vact,
                                                            const S* __restrict__ st, float* u,
                                                            const float* __restrict__ f, float* tmp, float* d,
                                                            const double* __restrict__ coef, int nsteps,
                                                            unsigned* bar, double* err, long spin_limit) {
    extern __shared__ float srow[];  // [RES_ROWS][ST_BS]
    __shared__ int s_ok;
    unsigned gen = 0;
    if (threadIdx.x == 0) gen = ld_acquire_u32(bar + 1);
    const int vx = nx + 1, vy = ny + 1, vz = nz + 1;
    const long nv = (long)vx * vy * vz;
    const long rs = StAddr<S>::stride(nv);
    const int tid = threadIdx.x, q = tid & 3;
    const long v = (blockIdx.x * (long)blockDim.x + tid) >> 2;
    const bool inb = v < nv;
    const bool act = inb && vact[v];
    const S* sb = st + StAddr<S>::base(inb ? v : 0);
    const int x = inb ? (int)(v % vx) : 0, y = inb ? (int)((v / vx) % vy) : 0,
              z = inb ? (int)(v / ((long)vx * vy)) : 0;
    long nj[7];
#pragma unroll
    for (int kk = 0; kk < 7; kk++) {
        const int k = q + 4 * kk;
        const int jx = x + k % 3 - 1, jy = y + (k / 3) % 3 - 1, jz = z + k / 9 - 1;
        const bool ok = act && k < 27 && jx >= 0 && jy >= 0 && jz >= 0 && jx < vx && jy < vy && jz < vz;
        nj[kk] = ok ? jx + (long)vx * (jy + (long)vy * jz) : (inb ? v : 0);
        const S* sk = sb + (long)(k * 9) * rs;
#pragma unroll
        for (int e = 0; e < 9; e++) {
            float a = 0.f;
            if (ok) {
                a = st_val(sk + e * rs);
                if (sizeof(S) == 2 && k == 13) a += st_val(sb + (243 + e) * rs);  // BF16 centre low part
            }
            srow[(kk * 9 + e) * ST_BS + tid] = a;
        }
    }
    // row q of the inverse centre block (scaled by 1 / det), f of the node, the direction d
    float i0 = 0.f, i1 = 0.f, i2 = 0.f, f0 = 0.f, f1 = 0.f, f2 = 0.f, dq = 0.f;
    if (act && q < 3) {
        float S9[9];
#pragma unroll
        for (int i = 0; i < 9; i++) S9[i] = st_centre<float>(sb, rs, i);
        const float a0 = S9[0], b0 = S9[1], c0 = S9[2], d0 = S9[3], e0 = S9[4], g0f = S9[5], g0 = S9[6], h0 = S9[7],
                    k0 = S9[8];
        const float A = e0 * k0 - g0f * h0, B = -(d0 * k0 - g0f * g0), Cc = d0 * h0 - e0 * g0;
        const float id = 1.f / (a0 * A + b0 * B + c0 * Cc);
        i0 = (q == 0 ? A : (q == 1 ? B : Cc)) * id;
        i1 = (q == 0 ? -(b0 * k0 - c0 * h0) : (q == 1 ? (a0 * k0 - c0 * g0) : -(a0 * h0 - b0 * g0))) * id;
        i2 = (q == 0 ? (b0 * g0f - c0 * e0) : (q == 1 ? -(a0 * g0f - c0 * d0) : (a0 * e0 - b0 * d0))) * id;
        f0 = f[v];
        f1 = f[nv + v];
        f2 = f[2 * nv + v];
    }
    __syncthreads();
    const long oq = (long)(q < 3 ? q : 0) * nv + (inb ? v : 0);
    for (int s = 0; s < nsteps; s++) {
        const float* src = (s & 1) ? tmp : u;
        float* dst = (s & 1) ? u : tmp;
        float Au[3] = {0.f, 0.f, 0.f};
#pragma unroll
        for (int kk = 0; kk < 7; kk++) {
            if (q + 4 * kk >= 27) break;
            const float u0 = __ldcg(src + nj[kk]), u1 = __ldcg(src + nv + nj[kk]), u2 = __ldcg(src + 2 * nv + nj[kk]);
#pragma unroll
            for (int r = 0; r < 3; r++)
                Au[r] += srow[(kk * 9 + 3 * r) * ST_BS + tid] * u0 + srow[(kk * 9 + 3 * r + 1) * ST_BS + tid] * u1 +
                         srow[(kk * 9 + 3 * r + 2) * ST_BS + tid] * u2;
        }
#pragma unroll
        for (int r = 0; r < 3; r++) {
            Au[r] += __shfl_xor_sync(0xffffffffu, Au[r], 1);
            Au[r] += __shfl_xor_sync(0xffffffffu, Au[r], 2);
        }
        if (inb && q < 3) {
            float res = 0.f, dn = 0.f;
            if (act) {
                const float zq = i0 * (f0 - Au[0]) + i1 * (f1 - Au[1]) + i2 * (f2 - Au[2]);
                dn = (s == 0 ? 0.f : (float)coef[2 * s] * dq) + (float)coef[2 * s + 1] * zq;
                res = __ldcg(src + oq) + dn;
            }
            dst[oq] = res;
            dq = dn;
        }
        if (s + 1 < nsteps || (nsteps & 1)) {
            if (!coop_grid_sync(bar, gen, &s_ok, spin_limit)) {
                if (threadIdx.x == 0) {
                    *err = 2.0;
                    u[0] = __int_as_float(0x7fc00000);
                }
                return;
            }
        }
    }
    if (inb && q < 3) {
        d[oq] = dq;
        if (nsteps & 1) u[oq] = __ldcg(tmp + oq);
    }
}

// ---------------------------------------------------------------------------
// Stencil kernel over the blocked FP32 / BF16 copies: the 31 KB (FP32) / 16 KB (BF16)
// stencil run of a 32-node block is fetched with one bulk asynchronous copy
// (cp.async.bulk, completion counted on an mbarrier) into a ring of NST shared-memory
// stages, so the stencil stream needs no registers in flight and the copies of the
// next blocks overlap the arithmetic of this one.  A CTA of 8 warps walks its blocks
// (blockIdx.x, + gridDim.x, ...): warp w sums the neighbours k = w, w+8, ... of the
// block's 32 nodes (lane = node, conflict-free stage reads), the eight partial sums
// meet in shared memory, and warps 0..2 finish component q = warp of every node.
// Every mbarrier wait is bounded: on a timeout the CTA waits (bounded) for its copies
// still in flight, writes NaN to the outputs it did not produce and sets the level's
// error slot, so the solve stops with an error instead of hanging.
// ---------------------------------------------------------------------------
constexpr int SB_BS = 256;
constexpr int SB_WARPS = SB_BS / 32;

template <typename S>
__host__ __device__ constexpr int sb_stages() { return sizeof(S) == 2 ? 4 : 3; }
template <typename T, typename S>
constexpr size_t sb_smem() {
    return 128 + (size_t)sb_stages<S>() * StAddr<S>::RS * 32 * sizeof(S) + SB_WARPS * 3 * 32 * sizeof(T);
}
template <typename S>
constexpr int sb_ctas_per_sm() { return sizeof(S) == 2 ? 3 : 2; }

template <typename T, int MODE, typename S>
__global__ void __launch_bounds__(SB_BS) k_st_bulk(int nx, int ny, int nz, const uint8_t* __restrict__ vact,
                                                    const S* __restrict__ st, const T* __restrict__ u,
                                                    const T* __restrict__ f, T* __restrict__ out, T* __restrict__ d,
                                                    T omega, const double* __restrict__ coef, int kstep,
                                                    double* __restrict__ errslot) {
    constexpr int RS = StAddr<S>::RS, NST = sb_stages<S>();
    constexpr uint32_t BLK_BYTES = RS * 32 * sizeof(S);
    constexpr long BLK_ELEMS = RS * 32;
    extern __shared__ __align__(128) unsigned char sm[];
    uint64_t* bar = reinterpret_cast<uint64_t*>(sm);
    S* stg = reinterpret_cast<S*>(sm + 128);
    T* red = reinterpret_cast<T*>(sm + 128 + NST * BLK_BYTES);
    T ca = T(0), cb = T(0);
    if (MODE == 3) {
        const double a_ = coef[2 * kstep], b_ = coef[2 * kstep + 1];
        ca = (T)a_;
        cb = (T)b_;
    }
    const int vx = nx + 1, vy = ny + 1, vz = nz + 1;
    const long nv = (long)vx * vy * vz;
    const long nblk = (nv + 31) / 32;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const long nmine = (long)blockIdx.x < nblk ? (nblk - 1 - blockIdx.x) / gridDim.x + 1 : 0;
    if (tid == 0) {
        for (int s = 0; s < NST; s++) rttc::mbar_init(&bar[s], 1);
        rttc::fence_mbar_init();
    }
    __syncthreads();
    // thread 0: the stencil run of this CTA's i-th block into stage i % NST
    auto issue = [&](long i) {
        const long b = blockIdx.x + i * (long)gridDim.x;
        uint64_t* br = &bar[i % NST];
        rttc::mbar_expect_tx(br, BLK_BYTES);
        rttc::bulk_g2s(stg + (i % NST) * BLK_ELEMS, st + b * BLK_ELEMS, BLK_BYTES, br);
    };
    if (tid == 0)
        for (long i = 0; i < NST - 1 && i < nmine; i++) issue(i);
    long i = 0, issued = nmine < NST - 1 ? nmine : NST - 1;
    bool ok = true;
    for (; i < nmine; i++) {
        // block i + NST - 1 goes into the stage block i - 1 used (released by the barrier ending iteration i - 1)
        if (issued < nmine) {
            if (tid == 0) issue(issued);
            issued++;
        }
        const int s = (int)(i % NST);
        const bool w = rttc::mbar_wait(&bar[s], (uint32_t)((i / NST) & 1));
        if (!__syncthreads_and(w)) {
            ok = false;
            break;
        }
        const S* sb = stg + s * BLK_ELEMS + lane;  // row j of this lane's node at sb[32 j]
        const long v = (blockIdx.x + i * (long)gridDim.x) * 32 + lane;
        const bool inb = v < nv;
        const bool act = inb && vact[v];
        T Au[3] = {T(0), T(0), T(0)};
        if (act) {
            const int x = (int)(v % vx), y = (int)((v / vx) % vy), z = (int)(v / ((long)vx * vy));
#pragma unroll
            for (int kk = 0; kk < 4; kk++) {
                const int k = warp + SB_WARPS * kk;
                if (k >= 27) break;
                const int jx = x + k % 3 - 1, jy = y + (k / 3) % 3 - 1, jz = z + k / 9 - 1;
                if (jx < 0 || jy < 0 || jz < 0 || jx >= vx || jy >= vy || jz >= vz) continue;
                const long nj = jx + (long)vx * (jy + (long)vy * jz);
                const T u0 = u[nj], u1 = u[nv + nj], u2 = u[2 * nv + nj];
                const S* sk = sb + k * 9 * 32;
#pragma unroll
                for (int r = 0; r < 3; r++) {
                    T a0 = (T)st_val(sk + (3 * r) * 32), a1 = (T)st_val(sk + (3 * r + 1) * 32),
                      a2 = (T)st_val(sk + (3 * r + 2) * 32);
                    if (sizeof(S) == 2 && k == 13) {
                        a0 += (T)st_val(sb + (243 + 3 * r) * 32);
                        a1 += (T)st_val(sb + (243 + 3 * r + 1) * 32);
                        a2 += (T)st_val(sb + (243 + 3 * r + 2) * 32);
                    }
                    Au[r] += a0 * u0 + a1 * u1 + a2 * u2;
                }
            }
        }
#pragma unroll
        for (int r = 0; r < 3; r++) red[(warp * 3 + r) * 32 + lane] = Au[r];
        __syncthreads();
        if (warp < 3 && inb) {
            const int q = warp;
            T A3[3];
#pragma unroll
            for (int r = 0; r < 3; r++) {
                A3[r] = red[r * 32 + lane];
#pragma unroll
                for (int w2 = 1; w2 < SB_WARPS; w2++) A3[r] += red[(3 * w2 + r) * 32 + lane];
            }
            const long oq = (long)q * nv + v;
            const T Aq = q == 0 ? A3[0] : (q == 1 ? A3[1] : A3[2]);
            if (MODE == 0) {
                out[oq] = act ? f[oq] - Aq : T(0);
            } else {
                T res = T(0), dn = T(0);
                if (act) {
                    T S9[9];
#pragma unroll
                    for (int e = 0; e < 9; e++) S9[e] = st_centre<T>(sb, 32, e);
                    const T a0 = S9[0], b0 = S9[1], c0 = S9[2], d0 = S9[3], e0 = S9[4], f0 = S9[5], g0 = S9[6],
                            h0 = S9[7], k0 = S9[8];
                    const T A = e0 * k0 - f0 * h0, B = -(d0 * k0 - f0 * g0), Cc = d0 * h0 - e0 * g0;
                    const T id = T(1) / (a0 * A + b0 * B + c0 * Cc);
                    const T i0 = q == 0 ? A : (q == 1 ? B : Cc);
                    const T i1 = q == 0 ? -(b0 * k0 - c0 * h0) : (q == 1 ? (a0 * k0 - c0 * g0) : -(a0 * h0 - b0 * g0));
                    const T i2 = q == 0 ? (b0 * f0 - c0 * e0) : (q == 1 ? -(a0 * f0 - c0 * d0) : (a0 * e0 - b0 * d0));
                    const T r0 = f[v] - A3[0], r1 = f[nv + v] - A3[1], r2 = f[2 * nv + v] - A3[2];
                    const T zq = (i0 * id) * r0 + (i1 * id) * r1 + (i2 * id) * r2;
                    if (MODE == 2) {
                        res = u[oq] + omega * zq;
                    } else {
                        dn = (kstep == 0 ? T(0) : ca * d[oq]) + cb * zq;
                        res = u[oq] + dn;
                    }
                }
                out[oq] = res;
                if (MODE == 3) d[oq] = dn;
            }
        }
        __syncthreads();  // the reduction buffer and stage s are free again
    }
    if (!ok) {
        for (long j = i; j < issued; j++) rttc::mbar_wait(&bar[j % NST], (uint32_t)((j / NST) & 1));
        if (tid == 0) errslot[0] = 1.0;
        for (long j = i; j < nmine; j++)
            for (int t = tid; t < 96; t += SB_BS) {
                const long v = (blockIdx.x + j * (long)gridDim.x) * 32 + (t & 31);
                if (v < nv) out[(long)(t >> 5) * nv + v] = T(NAN);
            }
    }
}

// ---------------------------------------------------------------------------
// The two coarsest levels of an FP32 cycle in one launch: smoothing from zero, residual, restriction, the coarsest
// product, prolongation and smoothing on the last smoothed level.  That level has a few thousand nodes at most, so a
// step is all launch and memory latency (3 us each, 20 of them per V-cycle with 8 smoothing steps); here one cluster
// of 16 blocks runs through them with a hardware cluster barrier in between.  Block b keeps the stencils of nodes
// [b npc, (b + 1) npc) in shared memory for the whole cycle (read through L1 from their usual place, every step cost
// as much as a launch), LPN lanes a node, with the node's inverse diagonal row and right-hand side in registers; the
// vectors, which other blocks write, go through L2 (ld.cg).  A PCG iteration of 97x61x45 (882 nodes, 8 steps)
// 279 -> 244 us, of 96x96x48 (1183 nodes) 344 -> 311 us.
// ---------------------------------------------------------------------------
constexpr int TC_CTAS = 16, TC_BS = 640;  // 640 threads: 96 registers, with 64 the products spill
constexpr long TC_MAX_N = 1300;  // rows of the coarsest inverse: 16 SMs read n^2 doubles (13 MB) in ~7 us
constexpr size_t TC_MAX_SMEM = 227 * 1024;

// lanes per node for npc nodes in a block, and the stride of a coefficient's nodes in shared memory: an odd multiple of
// the nodes in a warp, so that the LPN x 32 / LPN words of one load lie in 32 banks
__host__ __device__ constexpr int tc_lpn(int npc) { return npc <= TC_BS / 8 ? 8 : 4; }
__host__ __device__ constexpr int tc_stride(int npc, int lpn) {
    return ((npc + 32 / lpn - 1) / (32 / lpn) | 1) * (32 / lpn);
}
constexpr size_t tc_smem(int npc, long n) {
    return sizeof(float) * 243 * tc_stride(npc, tc_lpn(npc)) + sizeof(double) * n;
}

__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}

struct TailArgs {
    int vx, vy, vz, cvx, cvy, cvz;  // smoothed level, coarsest level
    int npc;                        // nodes of the smoothed level per block
    int na, npre, npost;
    bool cheby;
    float omega;
    const uint8_t *vact, *cvact;
    const float *st, *f;
    float *u, *r, *fc, *uc;
    const double *coef, *ainv;
    const int* aidx;
};

template <int LPN>
__global__ void __launch_bounds__(TC_BS) k_tail_cycle(const TailArgs a) {
    extern __shared__ double sd[];  // the coarsest right-hand side, then the block's stencils [243][stride]
    float* ss = reinterpret_cast<float*>(sd + 3 * a.na);
    const int tid = threadIdx.x, lane = tid & 31, q = tid % LPN, stride = tc_stride(a.npc, LPN);
    const int gid = blockIdx.x * TC_BS + tid;
    const int nv = a.vx * a.vy * a.vz, nvc = a.cvx * a.cvy * a.cvz;
    const int vb = blockIdx.x * a.npc, i = tid / LPN;  // the block's first node, the group's node in it
    const int v = i < a.npc && vb + i < nv ? vb + i : -1;
    const bool act = v >= 0 && a.vact[v];
    for (int c = tid / 32; c < 243; c += TC_BS / 32) {
        // 4-node pieces of a 128 B line
#pragma unroll 4
        for (int j = lane; j < a.npc; j += 32)
            if (vb + j < nv) ss[c * stride + j] = a.st[StAddr<float>::base(vb + j) + c * 32];
    }
    float f0 = 0.f, f1 = 0.f, f2 = 0.f, i0 = 0.f, i1 = 0.f, i2 = 0.f, dl = 0.f;
    if (act && q < 3) {
        f0 = __ldcg(a.f + v);
        f1 = __ldcg(a.f + nv + v);
        f2 = __ldcg(a.f + 2 * nv + v);
    }
    __syncthreads();
    if (act && q < 3) {
        float m[9];
#pragma unroll
        for (int k = 0; k < 9; k++) m[k] = ss[(117 + k) * stride + i];
        const float A = m[4] * m[8] - m[5] * m[7], B = m[5] * m[6] - m[3] * m[8], C = m[3] * m[7] - m[4] * m[6];
        const float id = 1.f / (m[0] * A + m[1] * B + m[2] * C);
        i0 = id * (q == 0 ? A : q == 1 ? B : C);
        i1 = id * (q == 0 ? m[2] * m[7] - m[1] * m[8] : q == 1 ? m[0] * m[8] - m[2] * m[6] : m[1] * m[6] - m[0] * m[7]);
        i2 = id * (q == 0 ? m[1] * m[5] - m[2] * m[4] : q == 1 ? m[2] * m[3] - m[0] * m[5] : m[0] * m[4] - m[1] * m[3]);
    }
    const int x = max(v, 0) % a.vx, y = max(v, 0) / a.vx % a.vy, z = max(v, 0) / (a.vx * a.vy);
    // A u of the group's node (every lane of it)
    auto product = [&](const float* src, float (&Au)[3]) {
        Au[0] = Au[1] = Au[2] = 0.f;
        if (act) {
            constexpr int NK = (27 + LPN - 1) / LPN;
#pragma unroll
            for (int k0 = 0; k0 < NK; k0 += 4) {  // 12 loads in flight
                float un[4][3];
#pragma unroll
                for (int kk = k0; kk < min(k0 + 4, NK); kk++) {
                    const int k = q + LPN * kk;
                    const int jx = x + k % 3 - 1, jy = y + (k / 3) % 3 - 1, jz = z + k / 9 - 1;
                    const bool in = k < 27 && jx >= 0 && jy >= 0 && jz >= 0 && jx < a.vx && jy < a.vy && jz < a.vz;
                    const int nj = jx + a.vx * (jy + a.vy * jz);
#pragma unroll
                    for (int c = 0; c < 3; c++) un[kk - k0][c] = in ? __ldcg(src + c * nv + nj) : 0.f;
                }
#pragma unroll
                for (int kk = k0; kk < min(k0 + 4, NK); kk++) {
                    const int k = q + LPN * kk;
                    if (k >= 27) break;
                    const float* s = ss + k * 9 * stride + i;
#pragma unroll
                    for (int r = 0; r < 3; r++)
                        Au[r] += s[(3 * r) * stride] * un[kk - k0][0] + s[(3 * r + 1) * stride] * un[kk - k0][1] +
                                 s[(3 * r + 2) * stride] * un[kk - k0][2];
                }
            }
        }
#pragma unroll
        for (int r = 0; r < 3; r++)
#pragma unroll
            for (int o = 1; o < LPN; o <<= 1) Au[r] += __shfl_xor_sync(0xffffffffu, Au[r], o);
    };
    // smoothing step k, src -> dst; from zero: src is not read
    auto smooth = [&](int k, const float* src, float* dst, bool zero) {
        const float ca = a.cheby ? (float)a.coef[2 * k] : 0.f, cb = a.cheby ? (float)a.coef[2 * k + 1] : a.omega;
        float Au[3] = {0.f, 0.f, 0.f};
        if (!zero) product(src, Au);
        if (v >= 0 && q < 3) {
            float res = 0.f;
            if (act) {
                const float zz = i0 * (f0 - Au[0]) + i1 * (f1 - Au[1]) + i2 * (f2 - Au[2]);
                const float old = zero ? 0.f : __ldcg(src + q * nv + v);
                dl = (k > 0 && a.cheby ? ca * dl : 0.f) + cb * zz;
                res = old + dl;
            }
            dst[q * nv + v] = res;
        }
        cluster_barrier();
    };
    // from zero the first step writes the vector that leaves the result in u
    const bool swap = a.npre % 2 == 1;
    for (int k = 0; k < a.npre; k++) {
        const bool even = (k % 2 == 0) != swap;
        smooth(k, even ? a.u : a.r, even ? a.r : a.u, k == 0);
    }
    {  // residual
        float Au[3];
        product(a.u, Au);
        if (v >= 0 && q < 3) a.r[q * nv + v] = act ? (q == 0 ? f0 - Au[0] : q == 1 ? f1 - Au[1] : f2 - Au[2]) : 0.f;
    }
    cluster_barrier();
    // restriction, 8 lanes per coarse node (as k_restrict2)
    for (int t0 = gid / 8; t0 < (nvc + TC_CTAS * TC_BS / 8 - 1) / (TC_CTAS * TC_BS / 8) * (TC_CTAS * TC_BS / 8);
         t0 += TC_CTAS * TC_BS / 8) {
        float s[3] = {0.f, 0.f, 0.f};
        if (t0 < nvc && a.cvact[t0]) {
            const int X = t0 % a.cvx, Y = t0 / a.cvx % a.cvy, Z = t0 / (a.cvx * a.cvy);
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const int k = (tid & 7) + 8 * i;
                if (k >= 27) break;
                const int dx = k % 3 - 1, dy = k / 3 % 3 - 1, dz = k / 9 - 1;
                const int fx = 2 * X + dx, fy = 2 * Y + dy, fz = 2 * Z + dz;
                if (fx < 0 || fy < 0 || fz < 0 || fx >= a.vx || fy >= a.vy || fz >= a.vz) continue;
                const int n = fx + a.vx * (fy + a.vy * fz);
                const float w = 0.125f * (float)((2 - abs(dx)) * (2 - abs(dy)) * (2 - abs(dz)));
                s[0] += w * __ldcg(a.r + n);
                s[1] += w * __ldcg(a.r + nv + n);
                s[2] += w * __ldcg(a.r + 2 * nv + n);
            }
        }
#pragma unroll
        for (int c = 0; c < 3; c++) {
            s[c] += __shfl_xor_sync(0xffffffffu, s[c], 1);
            s[c] += __shfl_xor_sync(0xffffffffu, s[c], 2);
            s[c] += __shfl_xor_sync(0xffffffffu, s[c], 4);
        }
        if (t0 < nvc && (tid & 7) < 3) a.fc[(tid & 7) * nvc + t0] = (tid & 7) == 0 ? s[0] : (tid & 7) == 1 ? s[1] : s[2];
    }
    cluster_barrier();
    // coarsest solve (as k_coarsest)
    const int n = 3 * a.na;
    for (int k = tid; k < a.na; k += TC_BS) {
        const int vc = a.aidx[k];
        sd[3 * k] = (double)__ldcg(a.fc + vc);
        sd[3 * k + 1] = (double)__ldcg(a.fc + nvc + vc);
        sd[3 * k + 2] = (double)__ldcg(a.fc + 2 * nvc + vc);
    }
    for (int vc = gid; vc < nvc; vc += TC_CTAS * TC_BS)
        if (!a.cvact[vc]) a.uc[vc] = a.uc[nvc + vc] = a.uc[2 * nvc + vc] = 0.f;
    __syncthreads();
    for (int k = gid / 32; k < n; k += TC_CTAS * TC_BS / 32) {
        const double* row = a.ainv + (long)k * n;
        double s[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        for (int j0 = lane; j0 < n; j0 += 256) {
            double b[8];
#pragma unroll
            for (int k = 0; k < 8; k++) b[k] = j0 + 32 * k < n ? row[j0 + 32 * k] : 0.0;
#pragma unroll
            for (int k = 0; k < 8; k++)
                if (j0 + 32 * k < n) s[k] += b[k] * sd[j0 + 32 * k];
        }
        double t = ((s[0] + s[1]) + (s[2] + s[3])) + ((s[4] + s[5]) + (s[6] + s[7]));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
        if (lane == 0) a.uc[(k % 3) * nvc + a.aidx[k / 3]] = (float)t;
    }
    cluster_barrier();
    // prolongation to the group's node
    if (act && q < 3) {
        const int ox = x & 1, oy = y & 1, oz = z & 1;
        const int c = x / 2 + a.cvx * (y / 2 + a.cvy * (z / 2));
        float s = 0.f;
#pragma unroll
        for (int k = 0; k < 8; k++) {
            const int bx = k & 1, by = (k >> 1) & 1, bz = k >> 2;
            const int w = (bx ? ox : 2 - ox) * (by ? oy : 2 - oy) * (bz ? oz : 2 - oz);
            // a corner without a weight may lie outside the coarse box
            if (w != 0) s += 0.125f * (float)w * __ldcg(a.uc + q * nvc + c + bx + a.cvx * (by + a.cvy * bz));
        }
        a.u[q * nv + v] = __ldcg(a.u + q * nv + v) + s;
    }
    cluster_barrier();
    for (int k = 0; k < a.npost; k++) smooth(k, k % 2 == 0 ? a.u : a.r, k % 2 == 0 ? a.r : a.u, false);
    // the last step wrote r: every lane copies what it wrote
    if (a.npost % 2 == 1 && v >= 0 && q < 3) a.u[q * nv + v] = __ldcg(a.r + q * nv + v);
}

// smoother copies of level stencils (layout above); one thread per (node, row group)
__global__ void k_st_to_f32(long nv, long nvpad, const double* __restrict__ st, float* __restrict__ out) {
    const long n = nvpad * 243;
    for (long o = blockIdx.x * (long)blockDim.x + threadIdx.x; o < n; o += (long)gridDim.x * blockDim.x) {
        const long blk = o / (243 * 32);
        const int j = (int)((o / 32) % 243), l = (int)(o & 31);
        const long v = blk * 32 + l;
        out[o] = v < nv ? (float)st[(long)j * nv + v] : 0.f;
    }
}

__device__ __forceinline__ uint16_t bf16_bits(double x) { return __bfloat16_as_ushort(__double2bfloat16(x)); }

// thread per (node, centre entry rc): the 26 off-centre entries of column rc are rounded, the
// centre entry takes their summed rounding error, stored as hi + lo
__global__ void k_st_to_bf16(long nv, long nvpad, const double* __restrict__ st, uint16_t* __restrict__ out) {
    const long n = nvpad * 9;
    for (long t = blockIdx.x * (long)blockDim.x + threadIdx.x; t < n; t += (long)gridDim.x * blockDim.x) {
        const long v = t % nvpad;
        const int rc = (int)(t / nvpad);
        uint16_t* ob = out + (v >> 5) * (252 * 32L) + (v & 31);
        if (v >= nv) {
            for (int k = 0; k < 27; k++) ob[(k * 9 + rc) * 32] = 0;
            ob[(243 + rc) * 32] = 0;
            continue;
        }
        double err = 0;
        for (int k = 0; k < 27; k++) {
            if (k == 13) continue;
            const double x = st[(long)(k * 9 + rc) * nv + v];
            const uint16_t b = bf16_bits(x);
            ob[(k * 9 + rc) * 32] = b;
            err += x - (double)__uint_as_float((uint32_t)b << 16);
        }
        const double c = st[(long)(117 + rc) * nv + v] + err;
        const uint16_t hi = bf16_bits(c);
        ob[(117 + rc) * 32] = hi;
        ob[(243 + rc) * 32] = bf16_bits(c - (double)__uint_as_float((uint32_t)hi << 16));
    }
}

// ---------------------------------------------------------------------------
// Ratio-4 restriction f_c(X) = sum_{|d| < 4} prod (4 - |d|)/4 * r_f(4X + d), one axis at a time.  A block of 128
// threads owns 31 x TY coarse columns of one component: a thread reads one fine column x, a fine plane's 4 TY + 3 rows
// go into TY row sums, those into the two coarse planes the fine plane touches, and a finished coarse plane is
// reduced along x through shared memory.  Each fine value is read 1.4 times (y and z overlap of neighbouring blocks,
// mostly L2 hits) instead of the 5.4 times, in 28-byte pieces, of a gather per coarse node.  511x256x256, FP32, the 23
// restrictions of a W-cycle: 740 -> 322 us with their launches.
// ---------------------------------------------------------------------------
constexpr int RS_CX = 31;  // coarse columns per block: 4 * 30 + 7 = 127 fine columns

template <typename T, int TY>
__global__ void __launch_bounds__(128) k_restrict4(int fvx, int fvy, int fvz, int cvx, int cvy, int cvz, int zcells,
                                                   const uint8_t* __restrict__ cvact, const T* __restrict__ rf,
                                                   T* __restrict__ fc) {
    __shared__ T row[TY][128];
    const int tid = threadIdx.x;
    const int nzb = (cvz + zcells - 1) / zcells, comp = blockIdx.z / nzb, zb = blockIdx.z - comp * nzb;
    const int X0 = blockIdx.x * RS_CX, Y0 = blockIdx.y * TY, Z0 = zb * zcells, Z1 = min(Z0 + zcells, cvz);
    const long fplane = (long)fvx * fvy, cplane = (long)cvx * cvy;
    rf += comp * fplane * fvz;
    fc += comp * cplane * cvz;
    const int x = 4 * X0 - 3 + tid, yb = 4 * Y0 - 3;
    const bool xok = x >= 0 && x < fvx && tid < 127;
    T cur[TY], nxt[TY];  // coarse planes Z and Z + 1
#pragma unroll
    for (int k = 0; k < TY; k++) cur[k] = nxt[k] = T(0);
    for (int Z = Z0; Z < Z1; Z++) {
        // the first plane of a chunk also needs the three fine planes below it
#pragma unroll 1
        for (int dz = Z == Z0 ? -3 : 0; dz < 4; dz++) {
            const int z = 4 * Z + dz;
            if (z < 0 || z >= fvz) continue;
            const T* p = rf + (long)z * fplane + (long)yb * fvx + x;
            T v[4 * TY + 3], acc[TY];
#pragma unroll
            for (int j = 0; j < 4 * TY + 3; j++) v[j] = xok && yb + j >= 0 && yb + j < fvy ? p[(long)j * fvx] : T(0);
#pragma unroll
            for (int k = 0; k < TY; k++) {
                acc[k] = v[4 * k + 3];
#pragma unroll
                for (int d = 1; d < 4; d++) acc[k] += T(0.25) * T(4 - d) * (v[4 * k + 3 - d] + v[4 * k + 3 + d]);
            }
            const T wc = T(0.25) * T(4 - abs(dz)), wn = dz > 0 ? T(0.25) * T(dz) : T(0);
#pragma unroll
            for (int k = 0; k < TY; k++) {
                cur[k] += wc * acc[k];
                nxt[k] += wn * acc[k];
            }
        }
#pragma unroll
        for (int k = 0; k < TY; k++) {
            row[k][tid] = cur[k];
            cur[k] = nxt[k];
            nxt[k] = T(0);
        }
        __syncthreads();
        for (int i = tid; i < TY * RS_CX; i += 128) {
            const int k = i / RS_CX, c = i - k * RS_CX;
            if (X0 + c < cvx && Y0 + k < cvy) {
                const T* q = &row[k][4 * c + 3];
                T s = q[0];
#pragma unroll
                for (int d = 1; d < 4; d++) s += T(0.25) * T(4 - d) * (q[-d] + q[d]);
                const long vc = X0 + c + (long)cvx * (Y0 + k) + cplane * Z;
                fc[vc] = cvact[vc] ? s : T(0);
            }
        }
        __syncthreads();
    }
}

// ratio-2 restriction on the stencil levels (27 taps), 8 lanes per coarse node: lane t sums taps t, t + 8, ...
template <typename T>
__global__ void __launch_bounds__(ST_BS) k_restrict2(int fvx, int fvy, int fvz, int cvx, int cvy, int cvz,
                                                     const uint8_t* __restrict__ cvact, const T* __restrict__ rf,
                                                     T* __restrict__ fc) {
    const long nvf = (long)fvx * fvy * fvz, nvc = (long)cvx * cvy * cvz;
    const int t = threadIdx.x & 7;
    const long ngroups = (long)gridDim.x * (blockDim.x >> 3);
    const long vend = ((nvc + ngroups - 1) / ngroups) * ngroups;
    for (long vc = (blockIdx.x * (long)blockDim.x + threadIdx.x) >> 3; vc < vend; vc += ngroups) {
        T s[3] = {T(0), T(0), T(0)};
        if (vc < nvc && cvact[vc]) {
            const int v32 = (int)vc, X = v32 % cvx, Y = v32 / cvx % cvy, Z = v32 / (cvx * cvy);
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const int k = t + 8 * i;
                if (k >= 27) break;
                const int dx = k % 3 - 1, dy = k / 3 % 3 - 1, dz = k / 9 - 1;
                const int x = 2 * X + dx, y = 2 * Y + dy, z = 2 * Z + dz;
                if (x < 0 || y < 0 || z < 0 || x >= fvx || y >= fvy || z >= fvz) continue;
                const long vf = x + (long)fvx * (y + (long)fvy * z);
                const T w = T(0.125) * T((2 - abs(dx)) * (2 - abs(dy)) * (2 - abs(dz)));
                s[0] += w * rf[vf];
                s[1] += w * rf[nvf + vf];
                s[2] += w * rf[2 * nvf + vf];
            }
        }
#pragma unroll
        for (int c = 0; c < 3; c++) {
            s[c] += __shfl_xor_sync(0xffffffffu, s[c], 1);
            s[c] += __shfl_xor_sync(0xffffffffu, s[c], 2);
            s[c] += __shfl_xor_sync(0xffffffffu, s[c], 4);
        }
        if (vc < nvc && t < 3) fc[(long)t * nvc + vc] = t == 0 ? s[0] : t == 1 ? s[1] : s[2];
    }
}

// u_f += trilinear interpolation of u_c.  A thread marches one fine column through zcells coarse cells, interpolating
// each coarse plane in x and y once (12 loads) for the R fine planes above and below it, where a thread per fine
// node gathered 24 coarse values.  511x256x256, FP32, the 23 prolongations of a W-cycle: 654 -> 396 us
// with their launches.
template <typename T, int R>
__global__ void __launch_bounds__(ST_BS) k_prolong(int fvx, int fvy, int fvz, int cvx, int cvy, int cvz, int zcells,
                                                   const uint8_t* __restrict__ fvact, const T* __restrict__ uc,
                                                   T* __restrict__ uf) {
    const int x = blockIdx.x * 32 + (threadIdx.x & 31), y = blockIdx.y * (ST_BS / 32) + (threadIdx.x >> 5);
    if (x >= fvx || y >= fvy) return;
    const long fplane = (long)fvx * fvy, cplane = (long)cvx * cvy, nvf = fplane * fvz, nvc = cplane * cvz;
    const int X = x / R, Y = y / R, ox = x - R * X, oy = y - R * Y;
    // the neighbouring coarse column and row only where they have a weight
    const long c00 = X + (long)cvx * Y, c10 = c00 + (ox ? 1 : 0), c01 = c00 + (oy ? cvx : 0), c11 = c01 + (ox ? 1 : 0);
    const T fx = T(ox) / T(R), fy = T(oy) / T(R);
    const T w00 = (T(1) - fx) * (T(1) - fy), w10 = fx * (T(1) - fy), w01 = (T(1) - fx) * fy, w11 = fx * fy;
    auto plane = [&](int Z, T (&p)[3]) {
        const T* q = uc + cplane * Z;
#pragma unroll
        for (int c = 0; c < 3; c++, q += nvc) p[c] = w00 * q[c00] + w10 * q[c10] + w01 * q[c01] + w11 * q[c11];
    };
    const int Z0 = blockIdx.z * zcells, Z1 = min(Z0 + zcells, cvz);
    T lo[3], hi[3];
    plane(Z0, lo);
    for (int Z = Z0; Z < Z1; Z++) {
        const bool up = Z + 1 < cvz;  // the last coarse plane has no fine plane above it
        if (up) plane(Z + 1, hi);
#pragma unroll
        for (int oz = 0; oz < R; oz++) {
            const int z = R * Z + oz;
            if (z >= fvz || (oz > 0 && !up)) break;
            const long v = x + (long)fvx * y + fplane * z;
            const bool act = fvact[v];
            const T f0 = uf[v], f1 = uf[nvf + v], f2 = uf[2 * nvf + v];
            if (act) {
                const T wh = T(oz) / T(R), wl = T(1) - wh;
                uf[v] = f0 + (oz ? wl * lo[0] + wh * hi[0] : lo[0]);
                uf[nvf + v] = f1 + (oz ? wl * lo[1] + wh * hi[1] : lo[1]);
                uf[2 * nvf + v] = f2 + (oz ? wl * lo[2] + wh * hi[2] : lo[2]);
            }
        }
#pragma unroll
        for (int c = 0; c < 3; c++) lo[c] = hi[c];
    }
}

// ---------------------------------------------------------------------------
// Galerkin assembly of the first coarse level directly from the elements: a coarse cell's matrix is
// M = sum_pos w_pos Q_pos, Q_pos = P_pos^T KE P_pos over its R^3 element positions, and the stencil of a node is the
// sum of its row blocks of the 8 cells around it.  k_galerkin_nodes computes it by nodes: the 8 corners of a cell
// partition the rows of M, so nothing is computed twice, and every stencil entry is written once, coalesced.  A block
// owns 32 x 2 nodes (x, y) of a layer with the weights of the 33 x 3 x 2 cells around them in shared memory; lane =
// node column, and a warp owns whole neighbours k (8 cell-neighbour pairs each), so that a Q block is loaded once for
// 64 nodes.  FP64 FMA bound (576 R^3 per node).  Elements touching a fixed node have weight 0 here and are added by
// k_galerkin_fixed.  160x144x96: 4.5 ms with cell matrices scattered through 8 colours, 0.5 ms here and 0.5 ms for the
// cells with fixed nodes.
// ---------------------------------------------------------------------------
constexpr int GN_BS = 256;

// neighbour k of warp w: the centre (8 cells), 2 faces (4 each), 4 edges (2 each), 8 corners (1 each); -1 ends a list
__constant__ int8_t GN_K[8][9] = {{13, -1, -1, -1, -1, -1, -1, -1, -1}, {4, 22, -1, -1, -1, -1, -1, -1, -1},
                                  {10, 16, -1, -1, -1, -1, -1, -1, -1}, {12, 14, -1, -1, -1, -1, -1, -1, -1},
                                  {1, 3, 5, 7, -1, -1, -1, -1, -1},     {9, 11, 15, 17, -1, -1, -1, -1, -1},
                                  {19, 21, 23, 25, -1, -1, -1, -1, -1}, {0, 2, 6, 8, 18, 20, 24, 26, -1}};

__device__ __forceinline__ double interp_w(int off, int corner, int R) {
    return (double)(R - abs(off - R * corner)) / (double)R;
}

// Qp: [corner m][corner n][pos][10] (9 entries of block (m, n) of Q_pos, one of padding)
template <int R>
__global__ void __launch_bounds__(GN_BS) k_galerkin_nodes(int fnx, int fny, int fnz, int cnx, int cny, int cnz,
                                                          const float* __restrict__ w, const double* __restrict__ Qp,
                                                          double* __restrict__ st) {
    constexpr int NP = R * R * R, CX = 33, CW = CX * 3 * 2;
    extern __shared__ double sw[];  // [NP][2 z][3 y][33 x]
    const int cvx = cnx + 1, cvy = cny + 1, cvz = cnz + 1;
    const long nvc = (long)cvx * cvy * cvz;
    const int X0 = blockIdx.x * 32, Y0 = blockIdx.y * 2, Z = blockIdx.z;
    for (int i = threadIdx.x; i < CX * R * 3 * R * 2 * R; i += GN_BS) {
        const int ix = i % (CX * R), iy = i / (CX * R) % (3 * R), iz = i / (CX * R * 3 * R);
        const int ex = R * (X0 - 1) + ix, ey = R * (Y0 - 1) + iy, ez = R * (Z - 1) + iz;
        double v = 0;
        if (ex >= 0 && ey >= 0 && ez >= 0 && ex < fnx && ey < fny && ez < fnz)
            v = fmaxf(w[ex + (long)fnx * (ey + (long)fny * ez)], 0.f);  // a NaN density is left to the solve to report
        const int pos = ix % R + R * (iy % R + R * (iz % R));
        sw[pos * CW + (iz / R * 3 + iy / R) * CX + ix / R] = v;
    }
    __syncthreads();
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    for (int li = 0; li < 8; li++) {
        const int k = GN_K[wid][li];
        if (k < 0) break;
        const int kx = k % 3 - 1, ky = k / 3 % 3 - 1, kz = k / 9 - 1;
        double acc[2][9];
#pragma unroll
        for (int q = 0; q < 9; q++) acc[0][q] = acc[1][q] = 0;
        for (int m = 0; m < 8; m++) {  // the node is corner m of the cell, its neighbour corner n
            const int nxb = (m & 1) + kx, nyb = ((m >> 1) & 1) + ky, nzb = (m >> 2) + kz;
            if (nxb < 0 || nxb > 1 || nyb < 0 || nyb > 1 || nzb < 0 || nzb > 1) continue;
            const double2* q2 = reinterpret_cast<const double2*>(Qp + ((m * 8 + nxb + 2 * nyb + 4 * nzb) * (long)NP) * 10);
            const double* wc = sw + ((1 - (m >> 2)) * 3 + 1 - ((m >> 1) & 1)) * CX + lane + 1 - (m & 1);
#pragma unroll 4
            for (int pos = 0; pos < NP; pos++) {
                const double2 a = q2[5 * pos], b = q2[5 * pos + 1], c = q2[5 * pos + 2], d = q2[5 * pos + 3],
                              e = q2[5 * pos + 4];
                const double w0 = wc[pos * CW], w1 = wc[pos * CW + CX];
                const double q[9] = {a.x, a.y, b.x, b.y, c.x, c.y, d.x, d.y, e.x};
#pragma unroll
                for (int t = 0; t < 9; t++) {
                    acc[0][t] += w0 * q[t];
                    acc[1][t] += w1 * q[t];
                }
            }
        }
#pragma unroll
        for (int j = 0; j < 2; j++) {
            if (X0 + lane >= cvx || Y0 + j >= cvy) continue;
            const long v = X0 + lane + (long)cvx * (Y0 + j + (long)cvy * Z);
#pragma unroll
            for (int t = 0; t < 9; t++) st[(long)(k * 9 + t) * nvc + v] = acc[j][t];
        }
    }
}

// the weights without the elements that touch a fixed node, and flags of the cells that hold such elements
template <int R>
__global__ void k_free_weights(int nx, int ny, int nz, int cnx, int cny, const float* __restrict__ w,
                               const uint8_t* __restrict__ vfix, float* __restrict__ wfree,
                               uint8_t* __restrict__ cfix) {
    const int vx = nx + 1, vy = ny + 1;
    const long ne = (long)nx * ny * nz;
    for (long e = blockIdx.x * (long)blockDim.x + threadIdx.x; e < ne; e += (long)gridDim.x * blockDim.x) {
        const int x = (int)(e % nx), y = (int)((e / nx) % ny), z = (int)(e / ((long)nx * ny));
        const long v = x + (long)vx * (y + (long)vy * z);
        bool fx = false;
#pragma unroll
        for (int j = 0; j < 8; j++) fx |= vfix[v + (j & 1) + (j & 2 ? vx : 0) + (j & 4 ? (long)vx * vy : 0)] != 0;
        const float we = w[e];
        wfree[e] = fx ? 0.f : we;
        if (fx && we != 0.f) cfix[x / R + (long)cnx * (y / R + (long)cny * (z / R))] = 1;
    }
}

// adds the elements with fixed nodes in their Dirichlet form K' (grid/Grid.cu:465-490): rows and columns of fixed nodes
// dropped, 1e6 on the fixed diagonal; P^T K' P of an element is T = K' P, then P^T T, 8 terms per entry and step.  One
// parity colour of cells per launch, so that no two cells share a node; a block looks at GF_CELLS cells and leaves at
// once where none is flagged.
constexpr int GF_BS = 288;  // 2 entries of the 576-entry cell matrix per thread
constexpr int GF_CELLS = 4;

template <int R>
__global__ void __launch_bounds__(GF_BS) k_galerkin_fixed(int fnx, int fny, int fnz, int cnx, int cny, int cnz,
                                                          int color, const uint8_t* __restrict__ cfix,
                                                          const float* __restrict__ w,
                                                          const uint8_t* __restrict__ vfix,
                                                          const double* __restrict__ KEg, double* __restrict__ st) {
    __shared__ double T[576], sP[R * R * R][8][8];  // sP[pos][element vertex][cell corner]
    __shared__ int cell[GF_CELLS];
    const int fvx = fnx + 1, fvy = fny + 1;
    const int cvx = cnx + 1, cvy = cny + 1, cvz = cnz + 1;
    const long nvc = (long)cvx * cvy * cvz;
    const int px = color & 1, py = (color >> 1) & 1, pz = (color >> 2) & 1;
    const int ccx = (cnx - px + 1) / 2, ccy = (cny - py + 1) / 2, ccz = (cnz - pz + 1) / 2;
    const int ncells = ccx * ccy * ccz;
    if (threadIdx.x < GF_CELLS) {
        const int t = blockIdx.x * GF_CELLS + threadIdx.x;
        int cid = -1;
        if (t < ncells) {
            cid = px + 2 * (t % ccx) + cnx * (py + 2 * (t / ccx % ccy) + cny * (pz + 2 * (t / (ccx * ccy))));
            if (!cfix[cid]) cid = -1;
        }
        cell[threadIdx.x] = cid;
    }
    if (!__syncthreads_or(threadIdx.x < GF_CELLS && cell[threadIdx.x < GF_CELLS ? threadIdx.x : 0] >= 0)) return;
    for (int i = threadIdx.x; i < R * R * R * 64; i += GF_BS) {
        const int pos = i / 64, j = i / 8 % 8, m = i % 8;
        sP[pos][j][m] = interp_w(pos % R + (j & 1), m & 1, R) * interp_w(pos / R % R + ((j >> 1) & 1), (m >> 1) & 1, R) *
                        interp_w(pos / (R * R) + (j >> 2), m >> 2, R);
    }
    // the thread's entries (3 m + row) * 24 + 3 n + col, half 0 and 1
    int m[2], n[2], row[2], col[2];
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const int t = threadIdx.x + h * GF_BS;
        m[h] = t / 72;
        row[h] = t / 24 % 3;
        n[h] = t % 24 / 3;
        col[h] = t % 3;
    }
    for (int li = 0; li < GF_CELLS; li++) {
        const int cid = cell[li];
        if (cid < 0) continue;
        const int X = cid % cnx, Y = cid / cnx % cny, Z = cid / (cnx * cny);
        double acc[2] = {0, 0};
        for (int pos = 0; pos < R * R * R; pos++) {
            const int ex = R * X + pos % R, ey = R * Y + pos / R % R, ez = R * Z + pos / (R * R);
            if (ex >= fnx || ey >= fny || ez >= fnz) continue;
            const double pen = w[ex + (long)fnx * (ey + (long)fny * ez)];
            if (pen == 0) continue;
            unsigned fm = 0;
#pragma unroll
            for (int j = 0; j < 8; j++)
                fm |= (vfix[(ex + (j & 1)) + (long)fvx * ((ey + ((j >> 1) & 1)) + (long)fvy * (ez + (j >> 2)))] != 0) << j;
            if (fm == 0) continue;
            __syncthreads();
#pragma unroll
            for (int h = 0; h < 2; h++) {  // row 3 j + row of K' times column n of P, j = m[h]
                const int j = m[h];
                double s = 0;
                for (int k = 0; k < 8; k++) {
                    double kk = 0;
                    if ((fm >> j & 1) || (fm >> k & 1)) kk = j == k && row[h] == col[h] ? 1e6 : 0.0;
                    else kk = pen * KEg[(3 * j + row[h]) * 24 + 3 * k + col[h]];
                    s += kk * sP[pos][k][n[h]];
                }
                T[threadIdx.x + h * GF_BS] = s;
            }
            __syncthreads();
#pragma unroll
            for (int h = 0; h < 2; h++)
                for (int j = 0; j < 8; j++) acc[h] += sP[pos][j][m[h]] * T[(3 * j + row[h]) * 24 + 3 * n[h] + col[h]];
        }
        // corner m of the cell, neighbour k(n - m)
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int dx = (n[h] & 1) - (m[h] & 1), dy = ((n[h] >> 1) & 1) - ((m[h] >> 1) & 1), dz = (n[h] >> 2) - (m[h] >> 2);
            const int k = (dx + 1) + 3 * (dy + 1) + 9 * (dz + 1);
            const long vc = (X + (m[h] & 1)) + (long)cvx * ((Y + ((m[h] >> 1) & 1)) + (long)cvy * (Z + (m[h] >> 2)));
            st[(long)(k * 9 + row[h] * 3 + col[h]) * nvc + vc] += acc[h];
        }
    }
}

// A_c = P^T A_f P for a dyadic (ratio 2) level from the finer stencil.  A warp per coarse node and block entry: lane i
// takes fine node i of the node's 3^3 support, reads that node's 27 entries and restricts them along each axis to the
// 3^3 coarse neighbours (the weights of an axis depend on the lane's offset on it), then the lanes are summed.  A
// thread per coarse node and entry looped over 729 products with 27 candidates each: 500 us a level, 79 us here.
__global__ void __launch_bounds__(ST_BS) k_galerkin_dyadic(int fnx, int fny, int fnz, int cnx, int cny, int cnz,
                                                           const uint8_t* __restrict__ fvact,
                                                           const uint8_t* __restrict__ cvact,
                                                           const double* __restrict__ stf, double* __restrict__ stc) {
    const int fvx = fnx + 1, fvy = fny + 1, fvz = fnz + 1;
    const int cvx = cnx + 1, cvy = cny + 1, cvz = cnz + 1;
    const long nvf = (long)fvx * fvy * fvz, nvc = (long)cvx * cvy * cvz;
    const int lane = threadIdx.x & 31;
    const int d[3] = {lane % 3 - 1, lane / 3 % 3 - 1, lane / 9 - 1};
    // weight of fine offset e = d + j - 1 in coarse neighbour s - 1: 1 - |2 (s - 1) - e| / 2 where positive
    double wt[3][3][3];
#pragma unroll
    for (int ax = 0; ax < 3; ax++)
#pragma unroll
        for (int j = 0; j < 3; j++)
#pragma unroll
            for (int q = 0; q < 3; q++) {
                const int g = abs(2 * (q - 1) - (d[ax] + j - 1));
                wt[ax][j][q] = g < 2 ? 0.5 * (2 - g) : 0.0;
            }
    const double wi = (d[0] ? 0.5 : 1.0) * (d[1] ? 0.5 : 1.0) * (d[2] ? 0.5 : 1.0);
    for (long t = (blockIdx.x * (long)blockDim.x + threadIdx.x) >> 5; t < nvc * 9; t += (long)gridDim.x * (ST_BS / 32)) {
        const long vc = t / 9;
        const int rc = (int)(t - vc * 9);
        const int X = (int)(vc % cvx), Y = (int)((vc / cvx) % cvy), Z = (int)(vc / ((long)cvx * cvy));
        double b[27];
#pragma unroll
        for (int j = 0; j < 27; j++) b[j] = 0;
        const int x = 2 * X + d[0], y = 2 * Y + d[1], z = 2 * Z + d[2];
        if (lane < 27 && cvact[vc] && x >= 0 && y >= 0 && z >= 0 && x < fvx && y < fvy && z < fvz) {
            const long vn = x + (long)fvx * (y + (long)fvy * z);
            if (fvact[vn]) {
#pragma unroll
                for (int j = 0; j < 27; j++) {
                    const int mx = x + j % 3 - 1, my = y + j / 3 % 3 - 1, mz = z + j / 9 - 1;
                    if (mx >= 0 && my >= 0 && mz >= 0 && mx < fvx && my < fvy && mz < fvz)
                        b[j] = stf[(long)(j * 9 + rc) * nvf + vn] * wi;
                }
#pragma unroll
                for (int ax = 0, str = 1; ax < 3; ax++, str *= 3)
#pragma unroll
                    for (int l = 0; l < 9; l++) {
                        const int o = ax == 0 ? 3 * l : ax == 1 ? l % 3 + 9 * (l / 3) : l;
                        const double a0 = b[o], a1 = b[o + str], a2 = b[o + 2 * str];
#pragma unroll
                        for (int q = 0; q < 3; q++)
                            b[o + q * str] = wt[ax][0][q] * a0 + wt[ax][1][q] * a1 + wt[ax][2][q] * a2;
                    }
            }
        }
        double mine = 0;
#pragma unroll
        for (int q = 0; q < 27; q++) {
            double v = b[q];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            if (lane == q) mine = v;
        }
        if (lane < 27) stc[(long)(lane * 9 + rc) * nvc + vc] = mine;
    }
}

__global__ void k_d2f(long n, const double* __restrict__ a, float* __restrict__ b) {
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) b[i] = (float)a[i];
}


}  // namespace

namespace rtk {

// stencil kernels on level 1 (the ratio-4 level, by far the largest) report under their own
// name, so a profile separates them from the small levels below
#define LVL_NAME(lvl, f64, base) \
    ((lvl) == 1 ? ((f64) ? base "_f64_l1" : base "_f32_l1") : ((f64) ? base "_f64" : base "_f32"))

template <typename T>
static const T* stp(rt_level& L);
template <>
const double* stp<double>(rt_level& L) { return L.st; }
template <>
const float* stp<float>(rt_level& L) { return L.st32; }

// the FP32 level kernels: bulk-copy stencil kernel over the blocked FP32 (or BF16) copy
template <int MODE, typename S>
static int launch_bulk(rt_hier* h, int lvl, const char* name, const S* st, const float* u, const float* f, float* out,
                       float* d, double omega, const double* coef, int kstep) {
    rt_level& L = h->L[lvl];
    const long nblk = (L.nv + 31) / 32;
    const long cap = (long)h->ctx->sm_count * sb_ctas_per_sm<S>();
    const unsigned grid = (unsigned)(nblk < cap ? nblk : cap);
    return rt_launch(h->ctx, name, [&] {
        k_st_bulk<float, MODE, S><<<grid, SB_BS, sb_smem<float, S>(), h->ctx->stream>>>(
            L.nx, L.ny, L.nz, L.vact, st, u, f, out, d, (float)omega, coef, kstep, h->scal + RT_SCAL_ERR);
    });
}

// the direct-load kernel: a block per 32 nodes
template <typename T, int MODE, typename S>
static int launch_direct(rt_hier* h, int lvl, const char* name, const S* st, const T* u, const T* f, T* out, T* d,
                        double omega, const double* coef, int kstep) {
    rt_level& L = h->L[lvl];
    return rt_launch(h->ctx, name, [&] {
        k_st_tile<T, MODE, S><<<(unsigned)((L.nv + 31) / 32), 288, 0, h->ctx->stream>>>(
            L.vx, L.vy, L.vz, L.vact, st, u, f, out, d, (T)omega, coef, kstep);
    });
}

template <int MODE, typename S>
static int launch_f32(rt_hier* h, int lvl, const char* name, const S* st, const float* u, const float* f, float* out,
                      float* d, double omega, const double* coef, int kstep) {
    if (h->st_variant[sizeof(S) == 2 ? 1 : 0] == 1)
        return launch_bulk<MODE, S>(h, lvl, name, st, u, f, out, d, omega, coef, kstep);
    return launch_direct<float, MODE, S>(h, lvl, name, st, u, f, out, d, omega, coef, kstep);
}

template <typename T>
int st_residual(rt_hier* h, int lvl, const T* u, const T* f, T* r) {
    rt_level& L = h->L[lvl];
    if constexpr (sizeof(T) == 4)
        return launch_f32<0, float>(h, lvl, LVL_NAME(lvl, false, "st_residual"), L.st32, u, f, r, nullptr, 0.0,
                                    nullptr, 0);
    else
        return launch_direct<T, 0, T>(h, lvl, LVL_NAME(lvl, true, "st_residual"), L.st, u, f, r, nullptr, 0.0, nullptr, 0);
}

template <typename T>
int st_gs(rt_hier* h, int lvl, T* u, const T* f, bool backward) {
    rt_level& L = h->L[lvl];
    for (int cc = 0; cc < 8; cc++) {
        int col = backward ? 7 - cc : cc;
        long ncol = (long)((L.vx - (col & 1) + 1) / 2) * ((L.vy - ((col >> 1) & 1) + 1) / 2) *
                    ((L.vz - ((col >> 2) & 1) + 1) / 2);
        if (ncol == 0) continue;
        RT_CHECK(rt_launch(h->ctx, LVL_NAME(lvl, sizeof(T) == 8, "st_gs"), [&] {
            if (ncol * 4 > (long)h->ctx->sm_count * 512)
                k_st_gs<T, 4><<<grid_for(h->ctx, 4 * ncol, 128), 128, 0, h->ctx->stream>>>(
                    L.vx, L.vy, L.vz, col, backward, L.vact, stp<T>(L), u, f);
            else
                k_st_gs<T, 32><<<grid_for(h->ctx, 32 * ncol, 128), 128, 0, h->ctx->stream>>>(
                    L.vx, L.vy, L.vz, col, backward, L.vact, stp<T>(L), u, f);
        }));
    }
    return RT_OK;
}

// the FP32 smoother reads the BF16 stencil copy when rt_params.coarse_bf16 is set
template <typename T>
static bool use_bf16(rt_hier* h, rt_level& L) {
    return sizeof(T) == 4 && h->P.coarse_bf16 && L.st16;
}

template <typename T>
int st_jacobi(rt_hier* h, int lvl, const T* u, const T* f, T* unew, double omega) {
    rt_level& L = h->L[lvl];
    if constexpr (sizeof(T) == 4) {
        if (use_bf16<T>(h, L))
            return launch_f32<2, uint16_t>(h, lvl, lvl == 1 ? "st_jacobi_bf16_l1" : "st_jacobi_bf16", L.st16, u, f,
                                           unew, nullptr, omega, nullptr, 0);
        return launch_f32<2, float>(h, lvl, LVL_NAME(lvl, false, "st_jacobi"), L.st32, u, f, unew, nullptr, omega,
                                    nullptr, 0);
    } else {
        return launch_direct<T, 2, T>(h, lvl, LVL_NAME(lvl, true, "st_jacobi"), L.st, u, f, unew, nullptr, omega, nullptr, 0);
    }
}

template <typename T>
int st_cheby(rt_hier* h, int lvl, const T* u, const T* f, T* unew, T* d, const double* coef, int kstep) {
    rt_level& L = h->L[lvl];
    if constexpr (sizeof(T) == 4) {
        if (use_bf16<T>(h, L))
            return launch_f32<3, uint16_t>(h, lvl, lvl == 1 ? "st_cheby_bf16_l1" : "st_cheby_bf16", L.st16, u, f,
                                           unew, d, 0.0, coef, kstep);
        return launch_f32<3, float>(h, lvl, LVL_NAME(lvl, false, "st_cheby"), L.st32, u, f, unew, d, 0.0, coef,
                                    kstep);
    } else {
        return launch_direct<T, 3, T>(h, lvl, LVL_NAME(lvl, true, "st_cheby"), L.st, u, f, unew, d, 0.0, coef, kstep);
    }
}
template <typename T>
int st_smooth0(rt_hier* h, int lvl, const T* f, T* out, double omega, T* d, const double* coef) {
    rt_level& L = h->L[lvl];
    const unsigned g = grid_for(h->ctx, L.nv, 128);
    return rt_launch(h->ctx, sizeof(T) == 8 ? "st_smooth0_f64" : "st_smooth0_f32", [&] {
        cudaStream_t s = h->ctx->stream;
        if (use_bf16<T>(h, L)) {
            if constexpr (sizeof(T) == 4) {
                if (coef) k_st_diag<T, 3, uint16_t><<<g, 128, 0, s>>>(L.nv, L.vact, L.st16, f, out, d, T(0), coef);
                else k_st_diag<T, 2, uint16_t><<<g, 128, 0, s>>>(L.nv, L.vact, L.st16, f, out, d, (T)omega, nullptr);
            }
        } else if (coef) {
            k_st_diag<T, 3><<<g, 128, 0, s>>>(L.nv, L.vact, stp<T>(L), f, out, d, T(0), coef);
        } else {
            k_st_diag<T, 2><<<g, 128, 0, s>>>(L.nv, L.vact, stp<T>(L), f, out, d, (T)omega, nullptr);
        }
    });
}
template int st_smooth0<double>(rt_hier*, int, const double*, double*, double, double*, const double*);
template int st_smooth0<float>(rt_hier*, int, const float*, float*, double, float*, const double*);

// co-resident blocks per SM of the fused kernels (queried once per context): the streaming form
// in coop_blocks_per_sm, the resident form (RES_SMEM of shared memory per block) in res_blocks_per_sm
static int coop_blocks(rt_hier* h, bool resident = false) {
    rt_ctx* c = h->ctx;
    if (c->coop_blocks_per_sm < 0) {
        int coop = 0, nb = 0, nr = 0;
        cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, c->device);
        if (coop) {
            int a = 0, b = 0;
            if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&a, k_st_cheby_coop<float>, ST_BS, 0) == cudaSuccess &&
                cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k_st_cheby_coop<uint16_t>, ST_BS, 0) == cudaSuccess)
                nb = a < b ? a : b;
            a = b = 0;
            if (cudaFuncSetAttribute(k_st_cheby_res<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)RES_SMEM) ==
                    cudaSuccess &&
                cudaFuncSetAttribute(k_st_cheby_res<uint16_t>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)RES_SMEM) == cudaSuccess &&
                cudaOccupancyMaxActiveBlocksPerMultiprocessor(&a, k_st_cheby_res<float>, ST_BS, RES_SMEM) == cudaSuccess &&
                cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k_st_cheby_res<uint16_t>, ST_BS, RES_SMEM) ==
                    cudaSuccess)
                nr = a < b ? a : b;
        }
        cudaGetLastError();
        c->coop_blocks_per_sm = nb;
        c->res_blocks_per_sm = nr;
    }
    return resident ? c->res_blocks_per_sm : c->coop_blocks_per_sm;
}

bool st_cheby_fused_ok(rt_hier* h) { return coop_blocks(h) > 0; }

int st_cheby_fused(rt_hier* h, int lvl, float* u, const float* f, float* tmp, float* d, const double* coef,
                   int nsteps) {
    rt_level& L = h->L[lvl];
    const int nb = coop_blocks(h);
    if (nb <= 0) return rt_fail(h->ctx, RT_ECUDA, "the device cannot run the fused Chebyshev sweeps");
    if (nsteps < 1 || nsteps > RT_CHEBY_MAXK) return rt_fail(h->ctx, RT_EINVAL, "fused Chebyshev: 1..16 steps");
    // one 4-lane group per node: the resident form when all groups fit on the device at once,
    // else the streaming form over a node loop
    const long want = rt_blocks(4 * L.nv, ST_BS);
    const long cap = (long)nb * h->ctx->sm_count;
    const bool resident = !((h->cheby_stream >> lvl) & 1u) && want <= (long)coop_blocks(h, true) * h->ctx->sm_count;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(resident ? want : (want < cap ? want : cap)));
    cfg.blockDim = dim3(ST_BS);
    cfg.dynamicSmemBytes = resident ? RES_SMEM : 0;
    cfg.stream = h->ctx->stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    unsigned* bar = reinterpret_cast<unsigned*>(h->scal + RT_SCAL_GBAR + lvl);
    double* err = h->scal + RT_SCAL_ERR;
    const long spin = (long)h->ctx->wait_limit;
    const bool bf = use_bf16<float>(h, L);
    cudaError_t e = cudaSuccess;
    RT_CHECK(rt_launch(h->ctx, bf ? (lvl == 1 ? "st_cheby_fused_bf16_l1" : "st_cheby_fused_bf16")
                                  : LVL_NAME(lvl, false, "st_cheby_fused"),
                       [&] {
                           if (resident && bf)
                               e = cudaLaunchKernelEx(&cfg, k_st_cheby_res<uint16_t>, L.nx, L.ny, L.nz,
                                                      (const uint8_t*)L.vact, (const uint16_t*)L.st16, u, f, tmp, d,
                                                      coef, nsteps, bar, err, spin);
                           else if (resident)
                               e = cudaLaunchKernelEx(&cfg, k_st_cheby_res<float>, L.nx, L.ny, L.nz,
                                                      (const uint8_t*)L.vact, (const float*)L.st32, u, f, tmp, d,
                                                      coef, nsteps, bar, err, spin);
                           else if (bf)
                               e = cudaLaunchKernelEx(&cfg, k_st_cheby_coop<uint16_t>, L.nx, L.ny, L.nz,
                                                      (const uint8_t*)L.vact, (const uint16_t*)L.st16, u, f, tmp, d,
                                                      coef, nsteps, bar, err, spin);
                           else
                               e = cudaLaunchKernelEx(&cfg, k_st_cheby_coop<float>, L.nx, L.ny, L.nz,
                                                      (const uint8_t*)L.vact, (const float*)L.st32, u, f, tmp, d,
                                                      coef, nsteps, bar, err, spin);
                       }));
    if (e != cudaSuccess)
        return rt_fail(h->ctx, RT_ECUDA, "fused Chebyshev launch failed: %s", cudaGetErrorString(e));
    return RT_OK;
}

template int st_cheby<double>(rt_hier*, int, const double*, const double*, double*, double*, const double*, int);
template int st_cheby<float>(rt_hier*, int, const float*, const float*, float*, float*, const double*, int);

template <typename T>
int restrict_(rt_hier* h, int lvl, const T* rf, T* fc) {
    rt_level& F = h->L[lvl - 1];
    rt_level& Cc = h->L[lvl];
    return rt_launch(h->ctx, sizeof(T) == 8 ? "restrict_f64" : "restrict_f32", [&] {
        if (Cc.ratio == 4) {
            // coarse planes per block: 8 (7/32 of the fine planes read twice), fewer until the blocks fill the GPU
            const int bx = (Cc.vx + RS_CX - 1) / RS_CX, by = (Cc.vy + 3) / 4;
            int zc = 8;
            while (zc > 1 && 3L * bx * by * ((Cc.vz + zc - 1) / zc) < 8L * h->ctx->sm_count) zc /= 2;
            const int nzb = 3 * ((Cc.vz + zc - 1) / zc);
            if (zc > 1)
                k_restrict4<T, 4><<<dim3(bx, by, nzb), 128, 0, h->ctx->stream>>>(F.vx, F.vy, F.vz, Cc.vx, Cc.vy, Cc.vz,
                                                                                 zc, Cc.vact, rf, fc);
            else
                k_restrict4<T, 1><<<dim3(bx, Cc.vy, nzb), 128, 0, h->ctx->stream>>>(F.vx, F.vy, F.vz, Cc.vx, Cc.vy,
                                                                                    Cc.vz, zc, Cc.vact, rf, fc);
        } else {
            k_restrict2<T><<<grid_for(h->ctx, 8 * Cc.nv, ST_BS), ST_BS, 0, h->ctx->stream>>>(
                F.vx, F.vy, F.vz, Cc.vx, Cc.vy, Cc.vz, Cc.vact, rf, fc);
        }
    });
}

template <typename T>
int prolong_add(rt_hier* h, int lvl, const T* uc, T* uf) {
    rt_level& F = h->L[lvl];
    rt_level& Cc = h->L[lvl + 1];
    return rt_launch(h->ctx, sizeof(T) == 8 ? "prolong_f64" : "prolong_f32", [&] {
        const int bx = (F.vx + 31) / 32, by = (F.vy + ST_BS / 32 - 1) / (ST_BS / 32);
        int zc = 8;  // coarse cells per thread, fewer until the blocks fill the GPU
        while (zc > 1 && (long)bx * by * ((Cc.vz + zc - 1) / zc) < 8L * h->ctx->sm_count) zc /= 2;
        const dim3 grid(bx, by, (Cc.vz + zc - 1) / zc);
        if (Cc.ratio == 4)
            k_prolong<T, 4><<<grid, ST_BS, 0, h->ctx->stream>>>(F.vx, F.vy, F.vz, Cc.vx, Cc.vy, Cc.vz, zc, F.vact, uc, uf);
        else
            k_prolong<T, 2><<<grid, ST_BS, 0, h->ctx->stream>>>(F.vx, F.vy, F.vz, Cc.vx, Cc.vy, Cc.vz, zc, F.vact, uc, uf);
    });
}

// Q_pos = P_pos^T KE P_pos for every element position in a coarse cell, as [corner m][corner n][pos][10]
static int build_Q(rt_hier* h, int R, double** Qdev) {
    const int NP = R * R * R;
    std::vector<double> Qh((size_t)NP * 640);
    for (int pos = 0; pos < NP; pos++) {
        int a = pos % R, b = (pos / R) % R, c = pos / (R * R);
        double P[8][8];
        for (int j = 0; j < 8; j++) {
            int o[3] = {a + (j & 1), b + ((j >> 1) & 1), c + (j >> 2)};
            for (int m = 0; m < 8; m++) {
                int mm[3] = {m & 1, (m >> 1) & 1, m >> 2};
                double wv = 1;
                for (int t = 0; t < 3; t++) wv *= (double)(R - abs(o[t] - R * mm[t])) / R;
                P[j][m] = wv;
            }
        }
        for (int m = 0; m < 8; m++)
            for (int row = 0; row < 3; row++)
                for (int n = 0; n < 8; n++)
                    for (int col = 0; col < 3; col++) {
                        double s = 0;
                        for (int j = 0; j < 8; j++) {
                            if (P[j][m] == 0) continue;
                            for (int k = 0; k < 8; k++)
                                s += P[j][m] * h->KE[(3 * j + row) * 24 + 3 * k + col] * P[k][n];
                        }
                        Qh[((size_t)(m * 8 + n) * NP + pos) * 10 + 3 * row + col] = s;
                    }
    }
    RT_CUDA(h->ctx, cudaMalloc(Qdev, sizeof(double) * Qh.size()));
    RT_CUDA(h->ctx, cudaMemcpyAsync(*Qdev, Qh.data(), sizeof(double) * Qh.size(), cudaMemcpyHostToDevice,
                                    h->ctx->stream));
    return RT_OK;
}

static constexpr size_t gn_smem(int R) { return sizeof(double) * R * R * R * 33 * 3 * 2; }

int galerkin_from_elements(rt_hier* h) {
    rt_level& F = h->L[0];
    rt_level& Cc = h->L[1];
    const int R = Cc.ratio;
    if (h->Qgal == nullptr || h->Qgal_ratio != R) {
        if (h->Qgal) cudaFree(h->Qgal);
        h->Qgal = nullptr;
        RT_CHECK(build_Q(h, R, &h->Qgal));
        h->Qgal_ratio = R;
    }
    rt_ctx* c = h->ctx;
    const float* w = h->w;
    uint8_t* cfix = nullptr;
    if (h->has_support) {  // ftmp: element scratch of the filter
        if (!Cc.cfix) RT_CUDA(c, cudaMalloc(&Cc.cfix, (size_t)Cc.ne));
        cfix = Cc.cfix;
        RT_CUDA(c, cudaMemsetAsync(cfix, 0, (size_t)Cc.ne, c->stream));
        RT_CHECK(rt_launch(c, "galerkin_weights", [&] {
            const unsigned g = grid_for(c, F.ne, ST_BS);
            if (R == 4)
                k_free_weights<4><<<g, ST_BS, 0, c->stream>>>(F.nx, F.ny, F.nz, Cc.nx, Cc.ny, h->w, h->vfix, h->ftmp, cfix);
            else
                k_free_weights<2><<<g, ST_BS, 0, c->stream>>>(F.nx, F.ny, F.nz, Cc.nx, Cc.ny, h->w, h->vfix, h->ftmp, cfix);
        }));
        w = h->ftmp;
    }
    RT_CHECK(rt_launch(c, "galerkin_nodes", [&] {
        const dim3 g((Cc.vx + 31) / 32, (Cc.vy + 1) / 2, Cc.vz);
        if (R == 4)
            k_galerkin_nodes<4><<<g, GN_BS, gn_smem(4), c->stream>>>(F.nx, F.ny, F.nz, Cc.nx, Cc.ny, Cc.nz, w, h->Qgal, Cc.st);
        else
            k_galerkin_nodes<2><<<g, GN_BS, gn_smem(2), c->stream>>>(F.nx, F.ny, F.nz, Cc.nx, Cc.ny, Cc.nz, w, h->Qgal, Cc.st);
    }));
    if (!cfix) return RT_OK;
    for (int color = 0; color < 8; color++) {
        const long ccells = (long)((Cc.nx - (color & 1) + 1) / 2) * ((Cc.ny - ((color >> 1) & 1) + 1) / 2) *
                            ((Cc.nz - (color >> 2) + 1) / 2);
        if (ccells == 0) continue;
        RT_CHECK(rt_launch(c, "galerkin_fixed", [&] {
            const unsigned g = (unsigned)((ccells + GF_CELLS - 1) / GF_CELLS);
            if (R == 4)
                k_galerkin_fixed<4><<<g, GF_BS, 0, c->stream>>>(F.nx, F.ny, F.nz, Cc.nx, Cc.ny, Cc.nz, color, cfix, h->w,
                                                                h->vfix, h->KE_dev, Cc.st);
            else
                k_galerkin_fixed<2><<<g, GF_BS, 0, c->stream>>>(F.nx, F.ny, F.nz, Cc.nx, Cc.ny, Cc.nz, color, cfix, h->w,
                                                                h->vfix, h->KE_dev, Cc.st);
        }));
    }
    return RT_OK;
}

int galerkin_from_stencil(rt_hier* h, int lvl) {
    rt_level& F = h->L[lvl - 1];
    rt_level& Cc = h->L[lvl];
    return rt_launch(h->ctx, "galerkin_dyadic", [&] {
        k_galerkin_dyadic<<<grid_for(h->ctx, Cc.nv * 9 * 32, ST_BS), ST_BS, 0, h->ctx->stream>>>(
            F.nx, F.ny, F.nz, Cc.nx, Cc.ny, Cc.nz, F.vact, Cc.vact, F.st, Cc.st);
    });
}

// one cluster with smem bytes of dynamic shared memory per block
static cudaLaunchConfig_t tail_config(size_t smem, cudaStream_t stream, cudaLaunchAttribute* at) {
    at->id = cudaLaunchAttributeClusterDimension;
    at->val.clusterDim.x = TC_CTAS;
    at->val.clusterDim.y = at->val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(TC_CTAS);
    cfg.blockDim = dim3(TC_BS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cfg;
}

// the last smoothed level and the coarsest one in one launch (k_tail_cycle): FP32 Jacobi or Chebyshev cycles from zero
// whose level fits the cluster and whose coarsest inverse 16 SMs can read in the time of a launch of all of them
bool tail_cycle_ok(rt_hier* h, int lvl, int smoother, int pre) {
    const int nl = (int)h->L.size();
    if (!h->ctx->tail_cluster || lvl != nl - 2 || lvl < 1 || pre < 1 || h->P.coarse_bf16 || ((h->cheby_fused >> lvl) & 1u)) return false;
    if (smoother != RT_SMOOTH_JACOBI && smoother != RT_SMOOTH_CHEBY) return false;
    const long n = 3L * h->L[lvl + 1].na, npc = (h->L[lvl].nv + TC_CTAS - 1) / TC_CTAS;
    return npc <= TC_BS / 4 && n <= TC_MAX_N && tc_smem((int)npc, n) <= TC_MAX_SMEM;
}

int tail_cycle(rt_hier* h, int lvl, int smoother, int pre, int post, double omega, const double* coef) {
    rt_level &L = h->L[lvl], &Cc = h->L[lvl + 1];
    const int npc = (int)((L.nv + TC_CTAS - 1) / TC_CTAS);
    TailArgs a{L.vx, L.vy, L.vz, Cc.vx, Cc.vy, Cc.vz, npc, Cc.na, pre, post, smoother == RT_SMOOTH_CHEBY, (float)omega, L.vact,
               Cc.vact, L.st32, L.f32, L.u32, L.r32, Cc.f32, Cc.u32, coef, Cc.ainv, Cc.aidx};
    cudaLaunchAttribute at;
    const cudaLaunchConfig_t cfg = tail_config(tc_smem(npc, 3L * Cc.na), h->ctx->stream, &at);
    cudaError_t e = cudaSuccess;
    RT_CHECK(rt_launch(h->ctx, "tail_cycle_f32", [&] {
        if (tc_lpn(npc) == 8) e = cudaLaunchKernelEx(&cfg, k_tail_cycle<8>, a);
        else e = cudaLaunchKernelEx(&cfg, k_tail_cycle<4>, a);
    }));
    if (e != cudaSuccess) return rt_fail(h->ctx, RT_ECUDA, "cluster launch failed: %s", cudaGetErrorString(e));
    return RT_OK;
}

int d2f(rt_hier* h, long n, const double* a, float* b) {
    return rt_launch(h->ctx, "d2f", [&] { k_d2f<<<grid_for(h->ctx, n, 256), 256, 0, h->ctx->stream>>>(n, a, b); });
}

// dynamic shared-memory limits of the bulk-copy stencil kernels, set once per device
int init_stencil_kernels(rt_ctx* c) {
    cudaError_t e[6] = {
        cudaFuncSetAttribute(k_galerkin_nodes<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)gn_smem(4)),
        cudaFuncSetAttribute(k_st_bulk<float, 0, float>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)sb_smem<float, float>()),
        cudaFuncSetAttribute(k_st_bulk<float, 2, float>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)sb_smem<float, float>()),
        cudaFuncSetAttribute(k_st_bulk<float, 3, float>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)sb_smem<float, float>()),
        cudaFuncSetAttribute(k_st_bulk<float, 2, uint16_t>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)sb_smem<float, uint16_t>()),
        cudaFuncSetAttribute(k_st_bulk<float, 3, uint16_t>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)sb_smem<float, uint16_t>())};
    for (cudaError_t x : e)
        if (x != cudaSuccess) return rt_fail(c, RT_ECUDA, "stencil kernel attributes: %s", cudaGetErrorString(x));
    // a cluster of 16 is above the portable size: where it does not fit, the levels run in separate launches
    c->tail_cluster = true;
    for (auto k : {k_tail_cycle<8>, k_tail_cycle<4>}) {
        cudaLaunchAttribute at;
        cudaLaunchConfig_t cfg = tail_config(TC_MAX_SMEM, c->stream, &at);
        int n = 0;
        if (cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
            cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TC_MAX_SMEM) != cudaSuccess ||
            cudaOccupancyMaxActiveClusters(&n, k, &cfg) != cudaSuccess || n < 1) {
            cudaGetLastError();
            c->tail_cluster = false;
        }
    }
    return RT_OK;
}

// the FP32 (and, with rt_params.coarse_bf16, BF16) smoother copies of level lvl's stencils
int stencil_copies(rt_hier* h, int lvl) {
    rt_level& L = h->L[lvl];
    const long nvpad = (L.nv + 31) / 32 * 32;
    RT_CHECK(rt_launch(h->ctx, "stencil_f32", [&] {
        k_st_to_f32<<<grid_for(h->ctx, nvpad * 243, 256), 256, 0, h->ctx->stream>>>(L.nv, nvpad, L.st, L.st32);
    }));
    if (!h->P.coarse_bf16) return RT_OK;
    return rt_launch(h->ctx, "stencil_bf16", [&] {
        k_st_to_bf16<<<grid_for(h->ctx, nvpad * 9, 256), 256, 0, h->ctx->stream>>>(L.nv, nvpad, L.st, L.st16);
    });
}

template int st_residual<double>(rt_hier*, int, const double*, const double*, double*);
template int st_residual<float>(rt_hier*, int, const float*, const float*, float*);
template int st_gs<double>(rt_hier*, int, double*, const double*, bool);
template int st_gs<float>(rt_hier*, int, float*, const float*, bool);
template int st_jacobi<double>(rt_hier*, int, const double*, const double*, double*, double);
template int st_jacobi<float>(rt_hier*, int, const float*, const float*, float*, double);
template int restrict_<double>(rt_hier*, int, const double*, double*);
template int restrict_<float>(rt_hier*, int, const float*, float*);
template int prolong_add<double>(rt_hier*, int, const double*, double*);
template int prolong_add<float>(rt_hier*, int, const float*, float*);

}  // namespace rtk
