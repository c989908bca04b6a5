// Adjoint of the radiance-cache transport with respect to the lights' emission.
//
// The cache's fixed point (the quantity the reference's scene preparation converges to,
// prep_mesh.cuh:182-213, and that every frame of poc_gpu.cu:433-530 estimates) is, for a fixed
// set of K rays per point,
//
//     L_l = T (E_l G_l + L_l),   T[i, j] = A_j / K x (rays of point i that reach point j),
//
// with G_l the direct light of light l at unit emission (k_build, poc_gpu.cu:369-391) and E_l
// its emission.  For J = sum_i w_i sum_l L_l[i] the adjoint importance u = w + T^T u gives
//
//     dJ / dE_l = sum_j (T^T u)_j G_l[j] = sum_j (u_j - w_j) G_l[j],
//
// one transposed solve for all lights instead of one forward solve per light.  The rays come
// from Ops<NL>::frozen_hits; this file builds the transposed ray lists (CSR, deterministic
// order), runs the forward and adjoint Jacobi sweeps and reduces the gradient in FP64 with a
// fixed summation order, so a result does not depend on the GPU or on the run.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <cmath>

#include "rc_adjoint.h"

namespace rc {
namespace adj {

namespace {

constexpr int B = 256;
constexpr long long FOLLOW_RAYS = 1 << 21;          // rays from which the sweeps' counts are followed (a sweep of 10 us)
constexpr int SCAN_ITEMS = 8;                       // per thread
constexpr int SCAN_TILE = B * SCAN_ITEMS;           // 2048 per block

__device__ __forceinline__ unsigned warp_max(unsigned v) {
    for (int o = 16; o > 0; o >>= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// incoming-ray count per point, and the rays that do not count
__global__ void k_count(const int* __restrict__ hits, long long n, int* __restrict__ cnt, unsigned long long* back) {
    unsigned nb = 0;
    for (long long e = blockIdx.x * (long long)B + threadIdx.x; e < n; e += (long long)gridDim.x * B) {
        const int j = hits[e];
        if (j >= 0) atomicAdd(&cnt[j], 1);
        else ++nb;
    }
    for (int o = 16; o > 0; o >>= 1) nb += __shfl_xor_sync(0xffffffffu, nb, o);
    if ((threadIdx.x & 31) == 0 && nb) atomicAdd(back, (unsigned long long)nb);
}

// exclusive scan of one tile of SCAN_TILE ints (in place allowed: a block reads its whole
// tile into registers before writing); the tile's total goes to bsum[blockIdx.x]
__global__ void __launch_bounds__(B) k_scan_tile(const int* in, int* out, int n, int* bsum) {
    __shared__ int wsum[B / 32];
    const long long base = (long long)blockIdx.x * SCAN_TILE + (long long)threadIdx.x * SCAN_ITEMS;
    int v[SCAN_ITEMS], t = 0;
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; ++k) {
        v[k] = base + k < n ? in[base + k] : 0;
        t += v[k];
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int x = t;   // inclusive warp scan of the thread totals
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) wsum[warp] = x;
    __syncthreads();
    int wpre = 0, total = 0;
    for (int k = 0; k < B / 32; ++k) {
        if (k < warp) wpre += wsum[k];
        total += wsum[k];
    }
    int run = wpre + x - t;
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; ++k) {
        if (base + k < n) out[base + k] = run;
        run += v[k];
    }
    if (threadIdx.x == 0) bsum[blockIdx.x] = total;
}

__global__ void k_scan_add(int* out, int n, const int* boff) {
    const long long e = blockIdx.x * (long long)B + threadIdx.x;
    if (e < n) out[e] += boff[e / SCAN_TILE];
}

// every counted ray into its target's segment, in arrival order
__global__ void k_fill(const int* __restrict__ hits, long long n, const int* __restrict__ off, int* __restrict__ fill,
                       int* __restrict__ unordered) {
    for (long long e = blockIdx.x * (long long)B + threadIdx.x; e < n; e += (long long)gridDim.x * B) {
        const int j = hits[e];
        if (j >= 0) unordered[off[j] + atomicAdd(&fill[j], 1)] = (int)e;
    }
}

// the segment of every entry sorted by ray index (rank = entries of the segment with a smaller
// ray index; ray indices are unique), stored as the ray's source point.  The entry's segment is
// its ray's hit point.  17.3 M rays: 462 us with a search of the offsets and an atomic maximum per
// segment on one address, 221 us
__global__ void k_rank(const int* __restrict__ hits, const int* __restrict__ off, int Np, const int* __restrict__ unordered, int K, long long cap,
                       int* __restrict__ src, int* maxseg) {
    const long long total = off[Np];
    for (long long q = blockIdx.x * (long long)B + threadIdx.x; q < total && q < cap; q += (long long)gridDim.x * B) {
        const int e = unordered[q], j = hits[e];
        const int a = off[j], b = off[j + 1];
        int rank = 0;
        for (int t = a; t < b; ++t) rank += unordered[t] < e;
        src[a + rank] = e / K;
        if (q == a && b - a > *(volatile int*)maxseg) atomicMax(maxseg, b - a);   // (one address: few need the atomic)
    }
}

// per point: direct light summed over the lights (l ascending) and albedo; the first gathered
// values A_j (d_j + L_j) with L = 0.  With `em` (NL emissions, device), the direct light is
// sum_l em_l G_l from the unit-emission build AEu instead of the state's own.
__global__ void k_prep(const float* __restrict__ AE, const float* __restrict__ AEu, const float* __restrict__ em, int aes, int NL,
                       int Np, float2* __restrict__ da, float* __restrict__ g0) {
    const int j = blockIdx.x * B + threadIdx.x;
    if (j >= Np) return;
    const float* ae = AE + (size_t)aes * j;
    float d = 0.f;
    if (em) {
        const float* au = AEu + (size_t)aes * j;
        for (int l = 0; l < NL; ++l) d += em[l] * au[1 + l];
    } else {
        for (int l = 0; l < NL; ++l) d += ae[1 + l];
    }
    da[j] = make_float2(d, ae[0]);
    g0[j] = ae[0] * (d + 0.f);
}

// The value of point i from the previous sweep's gathered values, its counted rays in ray order.
// Hit lists are read four rays at a time when K is a multiple of 4 (rows of 16 K bytes stay 16-byte
// aligned).
__device__ __forceinline__ float fwd_value(const int* __restrict__ hits, int K, int i, const float* __restrict__ gin) {
    float sum = 0.f;
    const int* h = hits + (size_t)i * K;
    if ((K & 3) == 0) {
        const int4* h4 = reinterpret_cast<const int4*>(h);
        for (int r = 0; r < K / 4; ++r) {
            const int4 q = __ldg(h4 + r);
            const float a = q.x >= 0 ? __ldcg(gin + q.x) : 0.f, b = q.y >= 0 ? __ldcg(gin + q.y) : 0.f;
            const float c = q.z >= 0 ? __ldcg(gin + q.z) : 0.f, d = q.w >= 0 ? __ldcg(gin + q.w) : 0.f;
            if (q.x >= 0) sum += a;
            if (q.y >= 0) sum += b;
            if (q.z >= 0) sum += c;
            if (q.w >= 0) sum += d;
        }
    } else {
        for (int r = 0; r < K; ++r) {
            const int j = __ldg(h + r);
            if (j >= 0) sum += __ldcg(gin + j);
        }
    }
    return sum / (float)K;
}
// w_j + (A_j / K) sum over the rays reaching j, in ray order, of uin[source] (four sources fetched at
// a time)
__device__ __forceinline__ float bwd_value(const int* __restrict__ src, int a, int b, int K, float A, float w, const float* __restrict__ uin) {
    float sum = 0.f;
    int q = a;
    for (; q + 4 <= b; q += 4) {
        const int s0 = __ldg(src + q), s1 = __ldg(src + q + 1), s2 = __ldg(src + q + 2), s3 = __ldg(src + q + 3);
        const float x0 = __ldcg(uin + s0), x1 = __ldcg(uin + s1), x2 = __ldcg(uin + s2), x3 = __ldcg(uin + s3);
        sum += x0;
        sum += x1;
        sum += x2;
        sum += x3;
    }
    for (; q < b; ++q) sum += __ldcg(uin + __ldg(src + q));
    return w + A * sum / (float)K;
}
__device__ __forceinline__ bool differ(float a, float b) { return __float_as_uint(a) != __float_as_uint(b); }

// The sweeps write, besides the iterate, one bit per point, set when the value that the next sweep
// gathers is not the one this sweep gathered (a warp's 32 points are a word), and add up the bits.
// bits is null where nobody asks.
__device__ __forceinline__ void note_bits(bool changed, int i, int Np, uint32_t* __restrict__ bits, unsigned* __restrict__ count) {
    const unsigned m = __ballot_sync(0xffffffffu, changed);
    if ((threadIdx.x & 31) == 0 && i < Np) bits[i >> 5] = m;
    const int n = __syncthreads_count(changed);
    if (threadIdx.x == 0 && n) atomicAdd(count, (unsigned)n);
}

struct Fwd {   // a forward sweep: L_i from the previous sweep's g; writes L and the next sweep's g = A (d + L)
    const int* hits;
    const float2* da;
    const float *gin, *Lprev;
    float *Lout, *gout;
    uint32_t* bits;
    unsigned* count;
};
struct Bwd {   // an adjoint sweep
    const int *off, *src;
    const float2* da;
    const float *w, *uin;
    float* uout;
    uint32_t* bits;
    unsigned* count;
};
// Full sweeps: the first nf blocks forward, the others adjoint (the two do not depend on each other, and
// together they have one tail instead of two: 129 us where the launches of their own took 67 + 70).  chg (may be null): the sweeps' largest changes
// and values.
__global__ void __launch_bounds__(B, 8) k_sweep(const Fwd f, const Bwd a, int nf, int K, int Np, unsigned* chg) {
    const bool fwd = (int)blockIdx.x < nf;
    const int i = (fwd ? (int)blockIdx.x : (int)blockIdx.x - nf) * B + threadIdx.x;
    uint32_t* bits = fwd ? f.bits : a.bits;
    float v = 0.f, dv = 0.f;
    bool changed = false;
    if (i < Np) {
        if (fwd) {
            v = fwd_value(f.hits, K, i, f.gin);
            f.Lout[i] = v;
            const float2 x = f.da[i];
            const float g = x.y * (x.x + v);
            f.gout[i] = g;
            if (bits) changed = differ(g, f.gin[i]);
            dv = fabsf(v - f.Lprev[i]);
        } else {
            v = bwd_value(a.src, a.off[i], a.off[i + 1], K, a.da[i].y, a.w[i], a.uin);
            a.uout[i] = v;
            const float u = a.uin[i];
            changed = differ(v, u);
            dv = fabsf(v - u);
        }
    }
    if (bits) note_bits(changed, i, Np, bits, fwd ? f.count : a.count);
    if (chg) {   // change of the sweep, and the largest value (non-negative floats order as their bits)
        const unsigned x = warp_max(__float_as_uint(dv)), y = warp_max(__float_as_uint(fabsf(v)));
        if ((threadIdx.x & 31) == 0) {
            atomicMax(&chg[fwd ? 0 : 2], x);
            atomicMax(&chg[fwd ? 1 : 3], y);
        }
    }
}

// The same sweeps once few values still change.  A point none of whose gathered values changed in the
// last sweep keeps its value to the last bit.  k_touch marks the points that do gather a changed value
// (of a changed g_j the sources of the rays reaching j, of a changed u_i the points that its rays
// reach), at a cost that falls with the changes; the sweep recomputes those, copies the others, and
// leaves the marks cleared.  1.08 M points, K = 16: 9 to 30 us behind 3 to 17 us of marks, where a full
// sweep takes 67 (forward) or 70 us (adjoint): those are bound by the L1, which takes one random
// sector per clock and SM.  A lookup of the gathered values' bits in shared memory instead of the marks
// cost 43 and 64 us.
__global__ void __launch_bounds__(B) k_touch(const uint32_t* __restrict__ bits, int words, const int* __restrict__ off, const int* __restrict__ list,
                                             int K, uint32_t* __restrict__ marks) {
    // four lanes to a word of 32 points; point j's list is [off[j], off[j + 1]), or [j K, j K + K) without off
    const int t = blockIdx.x * B + threadIdx.x, wd = t >> 2;
    if (wd >= words) return;
    for (uint32_t m = bits[wd]; m; m &= m - 1u) {
        const int j = 32 * wd + __ffs((int)m) - 1;
        const int a = off ? off[j] : j * K, b = off ? off[j + 1] : a + K;
        for (int q = a + (t & 3); q < b; q += 4) {
            const int i = __ldg(list + q);
            if (i >= 0) atomicOr(marks + (i >> 5), 1u << (i & 31));
        }
    }
}
__global__ void __launch_bounds__(B) k_fwd_few(const Fwd f, int K, int Np, uint32_t* __restrict__ marks) {
    const int i = blockIdx.x * B + threadIdx.x;
    const uint32_t word = i < Np ? marks[i >> 5] : 0u;
    __syncwarp();
    if ((threadIdx.x & 31) == 0 && word) marks[i >> 5] = 0u;
    bool changed = false;
    if (i < Np) {
        const float g0 = f.gin[i];
        float v = f.Lprev[i], g = g0;
        if (word >> (i & 31) & 1u) {
            v = fwd_value(f.hits, K, i, f.gin);
            const float2 x = f.da[i];
            g = x.y * (x.x + v);
            changed = differ(g, g0);
        }
        f.Lout[i] = v;
        f.gout[i] = g;
    }
    note_bits(changed, i, Np, f.bits, f.count);
}
__global__ void __launch_bounds__(B) k_bwd_few(const Bwd a, int K, int Np, uint32_t* __restrict__ marks) {
    const int j = blockIdx.x * B + threadIdx.x;
    const uint32_t word = j < Np ? marks[j >> 5] : 0u;
    __syncwarp();
    if ((threadIdx.x & 31) == 0 && word) marks[j >> 5] = 0u;
    bool changed = false;
    if (j < Np) {
        const float u = a.uin[j];
        float v = u;
        if (word >> (j & 31) & 1u) {
            v = bwd_value(a.src, a.off[j], a.off[j + 1], K, a.da[j].y, a.w[j], a.uin);
            changed = differ(v, u);
        }
        a.uout[j] = v;
    }
    note_bits(changed, j, Np, a.bits, a.count);
}

// Column c < NL: sum_j (u_j - w_j) G_c[j]; column NL: sum_j w_j L_j.  Block x sums a fixed slice of
// points (thread-strided, then a fixed tree), so the order never changes; it takes COLS columns at
// once, so that a point's record is read once or twice and not once per column (17 columns of 1.08 M
// points: 309 -> 134 us).
constexpr int COLS = 6;
__global__ void __launch_bounds__(B) k_grad_part(const float* __restrict__ AEu, int aes, int NL, int Np, const float* __restrict__ u,
                                                 const float* __restrict__ w, const float* __restrict__ L, double* __restrict__ part) {
    __shared__ double sh[B];
    const int c0 = blockIdx.y * COLS;
    const long long per = ((long long)Np + gridDim.x - 1) / gridDim.x;
    const long long j0 = per * blockIdx.x, j1 = min((long long)Np, j0 + per);
    double s[COLS];
#pragma unroll
    for (int k = 0; k < COLS; ++k) s[k] = 0.0;
    for (long long j = j0 + threadIdx.x; j < j1; j += B) {
        const float uj = u[j], wj = w[j];
        const double d = (double)uj - (double)wj;
        const float* G = AEu + (size_t)aes * j + 1 + c0;
#pragma unroll
        for (int k = 0; k < COLS; ++k) {
            if (c0 + k < NL) s[k] += d * (double)G[k];
            else if (c0 + k == NL) s[k] += (double)wj * (double)L[j];
        }
    }
#pragma unroll
    for (int k = 0; k < COLS; ++k) {
        if (c0 + k > NL) break;
        __syncthreads();
        sh[threadIdx.x] = s[k];
        __syncthreads();
        for (int o = B / 2; o > 0; o >>= 1) {
            if (threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
            __syncthreads();
        }
        if (threadIdx.x == 0) part[(size_t)(c0 + k) * gridDim.x + blockIdx.x] = sh[0];
    }
}

__global__ void __launch_bounds__(B) k_grad_final(const double* __restrict__ part, int G, double* __restrict__ out) {
    __shared__ double sh[B];
    const int c = blockIdx.x;
    double s = 0.0;
    for (int k = threadIdx.x; k < G; k += B) s += part[(size_t)c * G + k];
    sh[threadIdx.x] = s;
    __syncthreads();
    for (int o = B / 2; o > 0; o >>= 1) {
        if (threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) out[c] = sh[0];
}

int blocks_for(long long n) { return (int)((n + B - 1) / B); }
int stride_blocks(long long n) { return (int)(std::min)((n + B - 1) / B, 152LL * 16); }

cudaError_t scan_exclusive(const int* in, int* out, int n, int* scratch, cudaStream_t st, long long& launches) {
    const int nb = (n + SCAN_TILE - 1) / SCAN_TILE;
    k_scan_tile<<<nb, B, 0, st>>>(in, out, n, scratch);
    ++launches;
    if (nb > 1) {
        cudaError_t e = scan_exclusive(scratch, scratch, nb, scratch + nb, st, launches);
        if (e != cudaSuccess) return e;
        k_scan_add<<<blocks_for(n), B, 0, st>>>(out, n, scratch);
        ++launches;
    }
    return cudaGetLastError();
}

// Whether recomputing a sweep's touched points alone is expected to take less than a full sweep of its
// direction, when `n` values still change and `before` changed a sweep earlier.  Nanoseconds, measured at 1.08 M
// points and K = 16: a full sweep 3.8e-3 a ray; the points that gather one of n values the same a ray; their marks
// 8e-3 an entry; the copies of the others 3.2e-3 a point; two launches more and a tail of its own.  Counts that
// still grow are not followed: they are three sweeps old, and an objective on a few points reaches all in five.
// (270 k points, K = 8, 512 weights, 8 sweeps: 535 us with a threshold of Np / 10 alone, 502 before the changes were followed.)
bool few_pays(unsigned n, unsigned before, int Np, int K) {
    if (n > before) return false;
    const double full = 3.8e-3 * Np * K, touched = 1.0 - std::pow(1.0 - (double)n / Np, K);
    return 5000.0 + 3.2e-3 * Np + 8e-3 * n * K + touched * full < 0.95 * full;
}

}  // namespace

size_t bit_words(int Np) { return ((size_t)Np + 31) / 32; }

size_t scan_scratch_ints(long long n) {
    size_t s = 0;
    while (n > 1) {
        n = (n + SCAN_TILE - 1) / SCAN_TILE;
        s += (size_t)n;
    }
    return s + 1;
}

cudaError_t build_transpose(const Bufs& b, int Np, int K, cudaStream_t st, long long& launches) {
    const long long n = (long long)Np * K;
    cudaError_t e;
    if ((e = cudaMemsetAsync(b.cnt, 0, sizeof(int) * ((size_t)Np + 1), st)) != cudaSuccess) return e;
    if ((e = cudaMemsetAsync(b.fill, 0, sizeof(int) * (size_t)Np, st)) != cudaSuccess) return e;
    if ((e = cudaMemsetAsync(b.stats, 0, sizeof(Stats), st)) != cudaSuccess) return e;
    k_count<<<stride_blocks(n), B, 0, st>>>(b.hits, n, b.cnt, &b.stats->back);
    if ((e = scan_exclusive(b.cnt, b.off, Np + 1, b.scratch, st, launches)) != cudaSuccess) return e;
    k_fill<<<stride_blocks(n), B, 0, st>>>(b.hits, n, b.off, b.fill, b.unordered);
    k_rank<<<stride_blocks(n), B, 0, st>>>(b.hits, b.off, Np, b.unordered, K, n, b.src, &b.stats->max_incoming);
    launches += 3;
    return cudaGetLastError();
}

cudaError_t solve(Bufs* bp, int Np, int K, int NL, int aes, const float* AE, const float* AEu, const float* em, int iters,
                  cudaStream_t st, long long& launches) {
    const Bufs& b = *bp;
    cudaError_t e;
    k_prep<<<blocks_for(Np), B, 0, st>>>(AE, AEu, em, aes, NL, Np, b.da, b.g[0]);
    if ((e = cudaMemsetAsync(b.L[0], 0, sizeof(float) * (size_t)Np, st)) != cudaSuccess) return e;
    if ((e = cudaMemcpyAsync(b.u[0], b.w, sizeof(float) * (size_t)Np, cudaMemcpyDeviceToDevice, st)) != cudaSuccess) return e;
    // The sweeps.  On large problems the host follows, two sweeps behind, how many values still change:
    // when they are few enough (few_pays) the sweeps look first what to recompute (with K = 16, 10 % changing
    // values leave a fifth of the points alone, 1 % leave 85 %), and once none changes in two counted
    // sweeps, both buffers hold the fixed point and the sweeps up to the last have nothing to change.
    // The last sweep is always a full one: it measures the change.
    const bool follow = (long long)Np * K >= FOLLOW_RAYS && iters > 4;
    const int words = (Np + 31) / 32, touch_blocks = blocks_for(4LL * words);
    if (follow && ((e = cudaMemsetAsync(b.counts, 0, 2 * sizeof(unsigned) * (size_t)iters, st)) != cudaSuccess ||
                   (e = cudaMemsetAsync(b.marks, 0, sizeof(uint32_t) * (size_t)words, st)) != cudaSuccess))
        return e;
    bool few[2] = {false, false}, still[2] = {false, false};
    for (int t = 0; t < iters; ++t) {
        const bool last = t == iters - 1;
        if (follow && t >= 4 && (t & 1) == 0 && !last) {
            // the counts of sweep t - 3 and before have been copied behind sweep t - 3
            if ((e = cudaEventSynchronize(b.seen[(t >> 1) & 1])) != cudaSuccess) return e;
            for (int k = 0; k < 2; ++k) {
                const unsigned n = b.host_counts[2 * (t - 3) + k], before = b.host_counts[2 * (t - 4) + k];
                still[k] = n == 0 && before == 0;
                few[k] = still[k] || few_pays(n, before, Np, K);
            }
        }
        unsigned* chg = last ? b.stats->chg : nullptr;
        uint32_t *bi0 = follow ? b.bits[0][t & 1] : nullptr, *bi1 = follow ? b.bits[1][t & 1] : nullptr;
        uint32_t *bo0 = follow ? b.bits[0][(t + 1) & 1] : nullptr, *bo1 = follow ? b.bits[1][(t + 1) & 1] : nullptr;
        unsigned *c0 = follow ? b.counts + 2 * t : nullptr, *c1 = follow ? c0 + 1 : nullptr;
        const Fwd f{b.hits, b.da, b.g[t & 1], b.L[t & 1], b.L[(t + 1) & 1], b.g[(t + 1) & 1], bo0, c0};
        const Bwd a{b.off, b.src, b.da, b.w, b.u[t & 1], b.u[(t + 1) & 1], bo1, c1};
        const int nb = blocks_for(Np), nf = last || !few[0] ? nb : 0, na = last || !few[1] ? nb : 0;
        if (nf + na) {
            k_sweep<<<nf + na, B, 0, st>>>(f, a, nf, K, Np, chg);
            ++launches;
        }
        if (!nf && !still[0]) {
            k_touch<<<touch_blocks, B, 0, st>>>(bi0, words, b.off, b.src, K, b.marks);
            k_fwd_few<<<nb, B, 0, st>>>(f, K, Np, b.marks);
            launches += 2;
        }
        if (!na && !still[1]) {
            k_touch<<<touch_blocks, B, 0, st>>>(bi1, words, nullptr, b.hits, K, b.marks);
            k_bwd_few<<<nb, B, 0, st>>>(a, K, Np, b.marks);
            launches += 2;
        }
        if (follow && (t & 1) && t + 3 < iters - 1) {   // read before sweep t + 3
            if ((e = cudaMemcpyAsync(b.host_counts + 2 * (t - 1), b.counts + 2 * (t - 1), 4 * sizeof(unsigned), cudaMemcpyDeviceToHost, st)) !=
                    cudaSuccess ||
                (e = cudaEventRecord(b.seen[((t + 3) >> 1) & 1], st)) != cudaSuccess)
                return e;
        }
    }
    bp->L_final = b.L[iters & 1];
    bp->u_final = b.u[iters & 1];
    k_grad_part<<<dim3(GRAD_BLOCKS, (NL + 1 + COLS - 1) / COLS), B, 0, st>>>(AEu, aes, NL, Np, bp->u_final, b.w, bp->L_final, b.part);
    k_grad_final<<<NL + 1, B, 0, st>>>(b.part, GRAD_BLOCKS, b.stats->out);
    launches += 3;   // with k_prep
    return cudaGetLastError();
}

}  // namespace adj
}  // namespace rc
