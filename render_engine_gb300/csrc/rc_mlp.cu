// Learned radiance cache on the fifth-generation tensor cores (include/rc_mlp.h).
//
// Every layer product runs as tcgen05.mma: bf16 operands staged in shared memory in the
// canonical no-swizzle K-major layout (rc_umma.cuh), FP32 accumulators in tensor memory read
// back with tcgen05.ld, one elected thread issuing the MMAs and an mbarrier signalled by
// tcgen05.commit.  Every wait is bounded; a wait that gives up sets the error flag, and the
// kernel still releases its tensor memory.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <string>
#include <type_traits>
#include <vector>

#include "../../include/rc_mlp.h"
#include "rc_internal.h"
#include "rc_umma.cuh"

namespace {

using namespace rc::umma;
using rc::launch_dependent;
using rc::pdl_release;
using rc::pdl_wait;

constexpr uint32_t WAIT_LIMIT = 1u << 24;
constexpr int TILE_M = 128;

// ---------------------------------------------------------------- one tile product
// D[128 x N] = A[128 x K] B[N x K]^T, bf16 in, FP32 out; 128 threads (one warpgroup).
__global__ void __launch_bounds__(128) k_tile_product(const uint16_t* __restrict__ A, const uint16_t* __restrict__ B,
                                                      float* __restrict__ D, int K, int N, unsigned* __restrict__ err) {
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ uint64_t mbar;
    __shared__ uint32_t tmem_base;
    uint8_t* sa = smem;
    uint8_t* sb = smem + (size_t)TILE_M * K * 2;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    // stage A and B in the K-major core-matrix layout
    for (int idx = tid; idx < TILE_M * K; idx += 128) {
        const int r = idx / K, k = idx % K;
        *reinterpret_cast<uint16_t*>(sa + kmajor_offset(r, k, K)) = A[idx];
    }
    for (int idx = tid; idx < N * K; idx += 128) {
        const int r = idx / K, k = idx % K;
        *reinterpret_cast<uint16_t*>(sb + kmajor_offset(r, k, K)) = B[idx];
    }
    fence_proxy_async();
    if (tid == 0) mbar_init(&mbar, 1);
    const uint32_t ncols = N <= 32 ? 32 : (N <= 64 ? 64 : (N <= 128 ? 128 : 256));
    if (warp == 0) tmem_alloc(&tmem_base, ncols);
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    const uint32_t tmem = tmem_base;
    if (tid == 0) {
        const uint32_t idesc = idesc_bf16_f32(TILE_M, N);
        const uint32_t a0 = smem_u32(sa), b0 = smem_u32(sb);
        for (int kk = 0; kk < K / 16; ++kk)
            mma_bf16(tmem, smem_desc(a0 + 256u * kk, 128u, 16u * K), smem_desc(b0 + 256u * kk, 128u, 16u * K), idesc, kk > 0);
        mma_commit(&mbar);
    }
    const bool ok = mbar_wait(&mbar, 0, WAIT_LIMIT);
    if (!ok && lane == 0) atomicOr(err, 1u);
    fence_after_sync();
    if (ok) {
        const int row = warp * 32 + lane;
        for (int c = 0; c < N; c += 16) {
            float v[16];
            tmem_ld16(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)c, v);
            tmem_wait_ld();
#pragma unroll
            for (int i = 0; i < 16; ++i) D[(size_t)row * N + c + i] = v[i];
        }
    }
    fence_before_sync();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem, ncols);
}

// The bounded wait on its own: an mbarrier of one expected arrival, which one thread provides
// or nobody does; one thread polls it at most `polls` times.
__global__ void k_wait_check(uint32_t polls, int arrive, unsigned* __restrict__ err) {
    __shared__ uint64_t mbar;
    if (threadIdx.x == 0) mbar_init(&mbar, 1);
    __syncwarp();
    if (arrive && threadIdx.x == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&mbar)) : "memory");
    __syncwarp();
    if (threadIdx.x == 0 && !mbar_wait(&mbar, 0, polls)) atomicOr(err, 1u);
}

// ---------------------------------------------------------------- the network
// 168 input features (padded to 176) -> 64 -> 64 -> 64 -> 64 -> 16 outputs (the first n_out
// used), ReLU between layers, no biases.  Weights live as FP32 masters with their Adam
// moments, and as bf16 tiles W_l (rows = outputs, K = inputs) in the K-major core-matrix layout the
// forward products read; the gradients that flow back read the same tiles with the other index as
// K (rc_umma.cuh).
constexpr int K0 = 176, HID = 64, OUTP = 16, NLAYER = 5;
__host__ __device__ constexpr int in_dim(int l) { return l == 0 ? K0 : HID; }
__host__ __device__ constexpr int out_dim(int l) { return l == NLAYER - 1 ? OUTP : HID; }
__host__ __device__ constexpr int master_off(int l) { return l == 0 ? 0 : HID * K0 + (l - 1) * HID * HID; }
constexpr int NWEIGHT = HID * K0 + 3 * HID * HID + OUTP * HID;   // 24,576
__host__ __device__ constexpr int wf_off(int l) { return 2 * master_off(l); }   // byte offset of W_l's tile
constexpr int WF_BYTES = 2 * NWEIGHT;                                           // 49,152

// Words beside the training state: why this step's gradients must not be applied; blocks that have read
// the state.
enum MlpWord { WD_FAILED = 0, WD_TICKET, WD_COUNT };
constexpr unsigned STEP_NONFINITE = 1u, STEP_GAVE_UP = 2u;   // a gradient is not finite; a wait gave up

struct MlpArgs {
    const uint8_t* wbf;        // bf16 weight tiles
    const float4* P;           // point position (xyz)
    const float4* N;           // point normal (xyz)
    const float4* aux;         // albedo, direct light of lights 0..2
    const float* target;       // training targets, tstride floats per sample
    int tstride;
    const int* idx;            // sample -> point (null: identity)
    int n;                     // samples (a multiple of 128 when training)
    float* out;                // inference output, ostride floats per sample
    int ostride;
    int n_out;
    float lo[3], inv_ext[3];   // encoding box
    float* dwpart;             // training: weight gradients of each CTA, NWEIGHT per CTA
    float* loss;               // training: sum of the relative L2 loss (for reporting)
    float loss_scale;          // 1 / (samples x n_out)
    const float* scale;        // training: the loss scale of this step (device, MlpState::SCALE)
    unsigned* words;           // training: MlpWord
    uint32_t polls;            // polls of a completion wait before it gives up
    unsigned* err;
};

__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&h);
}
__device__ __forceinline__ void st_bf16(uint8_t* base, uint32_t off, float v) {
    *reinterpret_cast<__nv_bfloat16*>(base + off) = __float2bfloat16_rn(v);
}

// The 168 input features of one point (the rest of the 176 are zero): frequency encodings of
// the position in the box (12 octaves) and of the normal (4 octaves), one-blob encodings of
// both (16 and 4 bins per axis), the raw position, normal, direct light of three lights,
// albedo and a constant.  Produced eight at a time (one 16-byte group of the K-major tile);
// emit(group, f) stores them.  Two threads share a point: half 0 produces groups 0..8 (the
// position octaves), half 1 groups 9..21 (about the same work).
struct EncIn { float4 P, N, X; };   // position, normal, (albedo, direct light)
__device__ __forceinline__ EncIn encode_load(const MlpArgs& a, int pt) { return {a.P[pt], a.N[pt], a.aux[pt]}; }
template <class Emit>
__device__ __forceinline__ void encode(const MlpArgs& a, const EncIn& in, int half, Emit&& emit) {
    const float4 P = in.P, Nn = in.N, X = in.X;
    const float p[3] = {fminf(fmaxf((P.x - a.lo[0]) * a.inv_ext[0], 0.f), 1.f), fminf(fmaxf((P.y - a.lo[1]) * a.inv_ext[1], 0.f), 1.f),
                        fminf(fmaxf((P.z - a.lo[2]) * a.inv_ext[2], 0.f), 1.f)};
    const float nv[3] = {Nn.x, Nn.y, Nn.z};
    float f[8];
    // Four octaves per group: sincosf at the first, then the double-angle identities
    // sin 2w = 2 sin w cos w, cos 2w = (cos w - sin w)(cos w + sin w).  Three doublings grow the
    // error of the exact pair by at most about 8x (a few 1e-7), far below the bf16 rounding of
    // the features.
    auto octaves = [&](float w) {
        sincosf(w, &f[0], &f[1]);
#pragma unroll
        for (int j = 1; j < 4; ++j) {
            const float s = f[2 * j - 2], c = f[2 * j - 1];
            f[2 * j] = 2.f * s * c;
            f[2 * j + 1] = (c - s) * (c + s);
        }
    };
    if (half == 0) {
#pragma unroll
        for (int ax = 0; ax < 3; ++ax) {   // features 24 ax .. 24 ax + 23: sin / cos of 2^o pi p
            float w = 3.14159265f * p[ax];
#pragma unroll
            for (int g = 0; g < 3; ++g, w *= 16.f) {
                octaves(w);
                emit(ax * 3 + g, f);
            }
        }
        return;
    }
#pragma unroll
    for (int ax = 0; ax < 3; ++ax) {   // 72 + 8 ax: sin / cos of 2^o pi n
        octaves(3.14159265f * nv[ax]);
        emit(9 + ax, f);
    }
#pragma unroll
    for (int ax = 0; ax < 3; ++ax) {   // 96 + 16 ax: one-blob of p, 16 bins
        const float bp = p[ax] * 16.f;
        for (int g = 0; g < 2; ++g) {
#pragma unroll
            for (int j = 0; j < 8; ++j) f[j] = fmaxf(0.f, 1.f - fabsf(bp - (8 * g + j + 0.5f)));
            emit(12 + 2 * ax + g, f);
        }
    }
    float nb[12];   // 144 + 4 ax: one-blob of n, 4 bins
#pragma unroll
    for (int ax = 0; ax < 3; ++ax) {
        const float bn = (nv[ax] * 0.5f + 0.5f) * 4.f;
#pragma unroll
        for (int j = 0; j < 4; ++j) nb[4 * ax + j] = fmaxf(0.f, 1.f - fabsf(bn - (j + 0.5f)));
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) f[j] = nb[j];
    emit(18, f);
    f[0] = nb[8]; f[1] = nb[9]; f[2] = nb[10]; f[3] = nb[11];
    f[4] = p[0]; f[5] = p[1]; f[6] = p[2]; f[7] = nv[0];          // 156..159
    emit(19, f);
    f[0] = nv[1]; f[1] = nv[2]; f[2] = X.y; f[3] = X.z; f[4] = X.w; f[5] = X.x; f[6] = 1.f; f[7] = 0.f;   // 160..167
    emit(20, f);
#pragma unroll
    for (int j = 0; j < 8; ++j) f[j] = 0.f;
    emit(21, f);
}

// Inference over tiles of 128 queries, one persistent CTA per SM over the tiles blockIdx.x,
// blockIdx.x + gridDim.x, ...: tile k of the CTA is encoded by encoder group k % 2 (256 threads, two
// per query) into that group's X0 buffer and taken through the layers by chain k % 4 (128 threads,
// one per query) with its own activation buffer and 64 tensor-memory columns.  A chain gives the X0
// buffer back as soon as the first layer's product has read it, so two of them keep four chains
// busy, and encoding, products and epilogues of up to six tiles run at once.
//
// Bound by instruction issue and the chains' latency together.  1,082,802 queries: 92 us; as four
// groups of 256 threads that each encoded a tile and then took it through the layers, 141 us.  One
// tile alone: 8.7 us.
constexpr int IN_CHAINS = 4, IN_ENCODERS = 2;
constexpr int IN_CHAIN_T = 128, IN_ENC_T = 256;
constexpr int IN_THREADS = IN_CHAINS * IN_CHAIN_T + IN_ENCODERS * IN_ENC_T;
constexpr int IS_X = WF_BYTES;                              // X0 buffers, 128 x 176
constexpr int IS_H = IS_X + IN_ENCODERS * 128 * K0 * 2;     // activation buffers, 128 x 64
constexpr size_t INFER_SMEM = (size_t)IS_H + IN_CHAINS * 128 * HID * 2;
static_assert(INFER_SMEM > 114 * 1024 && INFER_SMEM <= 226 * 1024, "one inference CTA per SM");
// named barriers: X0 full (one per chain), X0 empty (one per buffer), a chain's own
enum InferBar { IB_FULL = 1, IB_EMPTY = IB_FULL + IN_CHAINS, IB_CHAIN = IB_EMPTY + IN_ENCODERS };
static_assert(IN_THREADS <= 1024 && IB_CHAIN + IN_CHAINS <= 16, "threads and barriers of an inference CTA");

// 16 accumulator columns -> ReLU -> bf16, as two 16-byte pieces of a K-major tile
__device__ __forceinline__ void relu_pack(const float (&v)[16], uint4& lo4, uint4& hi4) {
    lo4.x = pack_bf16(fmaxf(v[0], 0.f), fmaxf(v[1], 0.f));
    lo4.y = pack_bf16(fmaxf(v[2], 0.f), fmaxf(v[3], 0.f));
    lo4.z = pack_bf16(fmaxf(v[4], 0.f), fmaxf(v[5], 0.f));
    lo4.w = pack_bf16(fmaxf(v[6], 0.f), fmaxf(v[7], 0.f));
    hi4.x = pack_bf16(fmaxf(v[8], 0.f), fmaxf(v[9], 0.f));
    hi4.y = pack_bf16(fmaxf(v[10], 0.f), fmaxf(v[11], 0.f));
    hi4.z = pack_bf16(fmaxf(v[12], 0.f), fmaxf(v[13], 0.f));
    hi4.w = pack_bf16(fmaxf(v[14], 0.f), fmaxf(v[15], 0.f));
}
__device__ __forceinline__ uint4 pack8(const float (&f)[8]) {
    return make_uint4(pack_bf16(f[0], f[1]), pack_bf16(f[2], f[3]), pack_bf16(f[4], f[5]), pack_bf16(f[6], f[7]));
}
__device__ __forceinline__ void bar_sync(int id, int n) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory"); }
__device__ __forceinline__ void bar_arrive(int id, int n) { asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(n) : "memory"); }

__global__ void __launch_bounds__(IN_THREADS) k_mlp_infer(const MlpArgs a) {
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ uint64_t mbar[IN_CHAINS];
    __shared__ volatile int gave_up[IN_CHAINS];
    __shared__ uint32_t tmem_base;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    for (int i = tid; i < WF_BYTES / 16; i += IN_THREADS) reinterpret_cast<uint4*>(smem)[i] = reinterpret_cast<const uint4*>(a.wbf)[i];
    if (tid < IN_CHAINS) {
        mbar_init(&mbar[tid], 1);
        gave_up[tid] = 0;
    }
    if (warp == 0) tmem_alloc(&tmem_base, 64u * IN_CHAINS);
    fence_proxy_async();
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    const int ntiles = (a.n + 127) / 128;
    const int count = (ntiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;   // tiles of this CTA
    auto first_row = [&](int k) { return ((int)blockIdx.x + k * (int)gridDim.x) * 128; };
    if (warp >= IN_CHAINS * IN_CHAIN_T / 32) {
        const int g = (tid - IN_CHAINS * IN_CHAIN_T) / IN_ENC_T, et = tid % IN_ENC_T, row = et & 127, half = et >> 7;
        uint8_t* sx = smem + IS_X + g * (128 * K0 * 2);
        auto inputs = [&](int k) {
            const int s = first_row(k) + row, q = s < a.n ? s : 0;
            return encode_load(a, a.idx ? a.idx[q] : q);
        };
        EncIn next = inputs(g < count ? g : 0);
        for (int k = g; k < count; k += IN_ENCODERS) {
            const EncIn in = next;
            if (k + IN_ENCODERS < count) next = inputs(k + IN_ENCODERS);
            if (k >= IN_ENCODERS) bar_sync(IB_EMPTY + g, IN_CHAIN_T + IN_ENC_T);
            encode(a, in, half, [&](int k8, const float (&f)[8]) {
                *reinterpret_cast<uint4*>(sx + kmajor_offset(row, 8 * k8, K0)) = pack8(f);
            });
            fence_proxy_async();
            bar_arrive(IB_FULL + k % IN_CHAINS, IN_CHAIN_T + IN_ENC_T);
        }
    } else {
        const int c = warp >> 2, quarter = warp & 3, row = quarter * 32 + lane;
        const uint32_t sm0 = smem_u32(smem), tmem = tmem_base + 64u * (uint32_t)c, acc = tmem + ((uint32_t)(quarter * 32) << 16);
        uint8_t* sh = smem + IS_H + c * (128 * HID * 2);
        uint32_t phase = 0;
        bool ok = true;
        // One warp of the chain watches the barrier, the others wait for it without issuing (all warps
        // polling took 229 us where this took 141).  A wait that gives up raises the error flag, and the
        // chain stores no more outputs (its warps read that behind the barrier).  The product in flight is
        // waited for once more, so that nothing is overwritten or freed under it; if that gives up too,
        // no more products are issued, and the chain goes on through its barriers, so that nobody waits for it.
        auto wait = [&]() {
            if (quarter == 0) {
                if (ok && !mbar_wait(&mbar[c], phase, a.polls)) {
                    gave_up[c] = 1;
                    atomicOr(a.err, 1u);
                    ok = mbar_wait(&mbar[c], phase, WAIT_LIMIT);
                }
                fence_before_sync();
            }
            phase ^= 1u;
            bar_sync(IB_CHAIN + c, IN_CHAIN_T);
            fence_after_sync();
        };
        auto issue = [&](uint32_t a0, uint32_t b0, auto kc, uint32_t idesc) {
            constexpr int K = decltype(kc)::value;
            if (quarter == 0 && lane == 0 && ok) {
#pragma unroll
                for (int kk = 0; kk < K / 16; ++kk)
                    mma_bf16(tmem, smem_desc(a0 + 256u * kk, 128u, 16u * K), smem_desc(b0 + 256u * kk, 128u, 16u * K), idesc, kk > 0);
                mma_commit(&mbar[c]);
            }
            __syncwarp();
        };
        for (int k = c; k < count; k += IN_CHAINS) {
            const int b = k % IN_ENCODERS, s = first_row(k) + row;
            bar_sync(IB_FULL + c, IN_CHAIN_T + IN_ENC_T);
            issue(sm0 + IS_X + b * (128 * K0 * 2), sm0, std::integral_constant<int, K0>{}, idesc_bf16_f32(128, HID));
            wait();
            if (k + IN_ENCODERS < count) bar_arrive(IB_EMPTY + b, IN_CHAIN_T + IN_ENC_T);
#pragma unroll 1
            for (int l = 1; l < NLAYER; ++l) {
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    float v[2][16];
                    tmem_ld16(acc + 32u * q, v[0]);
                    tmem_ld16(acc + 32u * q + 16u, v[1]);
                    tmem_wait_ld();
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        uint4 lo4, hi4;
                        relu_pack(v[h], lo4, hi4);
                        uint8_t* dst = sh + kmajor_offset(row, 32 * q + 16 * h, HID);
                        *reinterpret_cast<uint4*>(dst) = lo4;
                        *reinterpret_cast<uint4*>(dst + 128) = hi4;
                    }
                }
                fence_before_sync();
                fence_proxy_async();
                bar_sync(IB_CHAIN + c, IN_CHAIN_T);
                fence_after_sync();
                issue(smem_u32(sh), sm0 + wf_off(l), std::integral_constant<int, HID>{}, idesc_bf16_f32(128, out_dim(l)));
                wait();
            }
            float v[16];
            tmem_ld16(acc, v);
            tmem_wait_ld();
            if (s < a.n && !gave_up[c]) {
                float* o = a.out + (size_t)s * a.ostride;
#pragma unroll
                for (int j = 0; j < OUTP; ++j)
                    if (j < a.n_out) o[j] = v[j];
            }
            fence_before_sync();
            bar_sync(IB_CHAIN + c, IN_CHAIN_T);   // the accumulator has been read
            fence_after_sync();
        }
        fence_before_sync();
    }
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem_base, 64u * IN_CHAINS);
}

// 16-byte asynchronous copies global -> shared (no register staging)
__device__ __forceinline__ void cp_async16(void* sdst, const void* gsrc) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(sdst)), "l"(gsrc) : "memory");
}

// n MMAs along K from base descriptors that advance by astep / bstep bytes each: an addition to the
// start address field (shared memory ends below its 2^18), so the one issuing thread spends a few
// instructions per MMA.  Rolled, like the loops over the layers below: a tile runs this code a few
// times only, and unrolled the instruction fetches cost more than the loops (60 us a step, not 49).
__device__ __forceinline__ void mma_chain(uint32_t d, uint64_t adesc, uint32_t astep, uint64_t bdesc, uint32_t bstep, int n, uint32_t idesc,
                                          bool fresh) {
    uint32_t acc = fresh ? 0u : 1u;
#pragma unroll 1
    for (int kk = 0; kk < n; ++kk) {
        mma_bf16(d, adesc, bdesc, idesc, acc);
        adesc += astep >> 4;
        bdesc += bstep >> 4;
        acc = 1u;
    }
}

// One training step's forward and backward pass: one CTA per SM over the tiles blockIdx.x,
// blockIdx.x + gridDim.x, ... of 128 samples, in that order, each tile forward and then backward
// while its activations are in shared memory.
//
// Warps 0..7 are the chain: they take each product out of tensor memory, form the next operand and
// hand it over (row = sample; the two threads of a row split the columns).  One thread of warp 16
// issues the products as the operands arrive, so that no warp of the chain spends its time on
// that; warps 8..15 encode the next tile's features meanwhile, into the other of two X0 buffers.
// Layer l's forward product goes to columns TR_DA .. of the tensor memory and back to shared memory
// as H_{l+1} = bf16(ReLU).  Backward, for l = 4 .. 0:
//     dZ_{l-1} = (dZ_l W_l) masked by ReLU'(H_l)   (issued first, its result waited for)
//     dW_l += dZ_l^T A_l over the tile's samples   (issued behind it, runs during the epilogue)
// dZ_l is stored as its rows (samples) by columns (features); the first product reads it K-major, the
// second with the samples as K, M-major, and likewise A_l and W_l with the other index as K, so no
// transposed copy of anything is made.  (dZ_l^T has out_dim(l) rows of the 128 the instruction
// takes: the rows beyond read whatever follows in shared memory and land in lanes that nothing
// reads.)  The weight gradients stay in tensor memory across the CTA's tiles (columns tr_dw_col(l))
// and leave once, as the CTA's slot of dwpart; the tile order within a CTA and the number of CTAs
// are fixed, so the sums are reproducible.
//
// Buffers: dZ_3 has one of its own, then dZ_2, dZ_1, dZ_0 take the places of H_4, H_3, H_2, whose
// last readers (dW_4, dW_3, dW_2) come before the product that the epilogue has just waited for.
//
// Bound by the latency of the chain (nine products, each waited for and passed through registers) at
// one tile per SM: the weights, two X0 buffers and the activations take 222 KB.
// 65,536 samples (512 tiles, four rounds): 42 us, 7.6 us a tile; as a forward kernel that wrote
// activations and their transposes to global memory and a backward kernel that read them, 45 + 54 us.
// With the chain's first warp issuing the products it took 50 us.
constexpr int TR_CHAIN = 256;                        // threads of the chain
constexpr int TR_ENCODE = 256;                       // threads that encode
constexpr int TR_THREADS = TR_CHAIN + TR_ENCODE + 32;
constexpr uint32_t TR_COLS = 512, TR_DA = 448;
__host__ __device__ constexpr uint32_t tr_dw_col(int l) { return l == 0 ? 0u : (uint32_t)(K0 + (l - 1) * HID); }
static_assert(tr_dw_col(NLAYER - 1) + HID <= TR_DA && TR_DA + HID <= TR_COLS, "tensor-memory columns of a training step");
constexpr int TS_X = WF_BYTES;                       // X0, two buffers of 128 x 176
constexpr int TS_H = TS_X + 2 * 128 * K0 * 2;        // H_1 .. H_4, 128 x 64 each
constexpr int TS_E = TS_H + 4 * 128 * HID * 2;       // dZ_3
constexpr int TS_DY = TS_E + 128 * HID * 2;          // dZ_4, 128 x 16
constexpr int TS_END = TS_DY + 128 * OUTP * 2 + 2048;   // 2 KB that the rows beyond dZ_4^T's 16 may read
constexpr size_t TRAIN_SMEM = (size_t)TS_END;
static_assert(TRAIN_SMEM > 114 * 1024 && TRAIN_SMEM <= 226 * 1024, "one training CTA per SM, all of its tensor memory");
// named barriers: an operand handed over by the chain; an X0 buffer full, empty (one of each per buffer)
enum TrainBar { TB_CHAIN = 1, TB_FULL = 2, TB_EMPTY = 4 };

__global__ void __launch_bounds__(TR_THREADS) k_mlp_train(const MlpArgs a, int ntiles) {
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ uint64_t mbar;
    __shared__ volatile int gave_up, lost;
    __shared__ uint32_t tmem_base;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    constexpr int W_ENCODE = TR_CHAIN / 32, W_ISSUE = (TR_CHAIN + TR_ENCODE) / 32;
    pdl_release();
    if (tid == 0) {
        mbar_init(&mbar, 1);
        gave_up = lost = 0;
    }
    if (warp == W_ISSUE) tmem_alloc(&tmem_base, TR_COLS);
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    pdl_wait();   // the kernel before: the last step's weights, the caller's inputs
    const uint32_t tmem = tmem_base, sm0 = smem_u32(smem);
    const int count = (ntiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;   // tiles of this CTA
    auto hbuf = [](int l) { return (uint32_t)(TS_H + (l - 1) * (128 * HID * 2)); };
    auto xbuf = [](int it) { return (uint32_t)(TS_X + (it & 1) * (128 * K0 * 2)); };
    if (warp == W_ISSUE) {
        // the products, in the order of their operands; never waits for a product itself
        for (int it = 0; it < count; ++it) {
            if (it == 0) bar_sync(TB_CHAIN, TR_CHAIN + 32);   // the weights
            bar_sync(TB_FULL + (it & 1), TR_ENCODE + 32);
#pragma unroll 1
            for (int l = 0; l < NLAYER; ++l) {
                const bool stop = lost;   // (read while it would wait anyway; at most one product more is issued)
                if (l > 0) bar_sync(TB_CHAIN, TR_CHAIN + 32);
                fence_after_sync();
                if (lane == 0 && !stop) {
                    const uint32_t K = (uint32_t)in_dim(l);
                    mma_chain(tmem + TR_DA, smem_desc(sm0 + (l == 0 ? xbuf(it) : hbuf(l)), 128u, 16u * K), 256u,
                              smem_desc(sm0 + wf_off(l), 128u, 16u * K), 256u, (int)K / 16, idesc_bf16_f32(128, out_dim(l)), true);
                    mma_commit(&mbar);
                }
                __syncwarp();
            }
#pragma unroll 1
            for (int l = NLAYER - 1; l >= 0; --l) {
                const bool stop = lost;
                bar_sync(TB_CHAIN, TR_CHAIN + 32);
                fence_after_sync();
                if (lane == 0 && !stop) {
                    const uint32_t Kin = (uint32_t)in_dim(l), Nout = (uint32_t)out_dim(l);
                    const uint32_t z = sm0 + (l == 4 ? (uint32_t)TS_DY : (l == 3 ? (uint32_t)TS_E : hbuf(l + 2)));
                    if (l >= 1) {
                        mma_chain(tmem + TR_DA, smem_desc(z, 128u, 16u * Nout), 256u, smem_desc(sm0 + wf_off(l), 16u * HID, 128u), 32u * HID,
                                  (int)Nout / 16, idesc_bf16_f32(128, HID, false, true), true);
                        mma_commit(&mbar);
                    }
                    mma_chain(tmem + tr_dw_col(l), smem_desc(z, 16u * Nout, 128u), 32u * Nout,
                              smem_desc(sm0 + (l == 0 ? xbuf(it) : hbuf(l)), 16u * Kin, 128u), 32u * Kin, 8, idesc_bf16_f32(128, (int)Kin, true, true),
                              it == 0);
                    if (l == 0 && it == count - 1) mma_commit(&mbar);   // the last dW_0
                }
                __syncwarp();
            }
        }
    } else if (warp >= W_ENCODE) {
        const int et = tid - TR_CHAIN, row = et & 127, half = et >> 7;
        auto inputs = [&](int it) {
            const int s = ((int)blockIdx.x + it * (int)gridDim.x) * 128 + row;
            return encode_load(a, a.idx ? a.idx[s] : s);
        };
        EncIn next = inputs(0);
        for (int it = 0; it < count; ++it) {
            const EncIn in = next;
            uint8_t* sx = smem + xbuf(it);
            if (it + 1 < count) next = inputs(it + 1);
            if (it >= 2) bar_sync(TB_EMPTY + (it & 1), TR_CHAIN + TR_ENCODE);
            encode(a, in, half, [&](int k8, const float (&f)[8]) {
                *reinterpret_cast<uint4*>(sx + kmajor_offset(row, 8 * k8, K0)) = pack8(f);
            });
            fence_proxy_async();
            bar_arrive(TB_FULL + (it & 1), TR_ENCODE + 32);
        }
    } else {
        const int quarter = warp & 3, half = warp >> 2, row = quarter * 32 + lane;
        const uint32_t acc = tmem + TR_DA + ((uint32_t)(quarter * 32) << 16);
        uint32_t phase = 0;
        bool ok = true;
        // Every warp watches the barrier itself.  A wait that gives up raises the error flag and marks the
        // step failed: no gradients leave this CTA, and Adam leaves weights and state alone.  The product in
        // flight is waited for once more, so that nothing is overwritten or freed under it; if that gives up
        // too, no more products are issued, and the chain goes on through its barriers, so that nobody
        // waits for it.
        auto wait = [&]() {
            if (ok && !mbar_wait(&mbar, phase, a.polls)) {
                gave_up = 1;
                atomicOr(a.err, 1u);
                atomicOr(a.words + WD_FAILED, STEP_GAVE_UP);
                ok = mbar_wait(&mbar, phase, WAIT_LIMIT);
                if (!ok) lost = 1;
            }
            phase ^= 1u;
            fence_after_sync();
        };
        auto handover = [&]() {   // this thread's writes to shared memory, and its reads of the accumulator, before the next product
            fence_before_sync();
            fence_proxy_async();
            bar_arrive(TB_CHAIN, TR_CHAIN + 32);
        };
        for (int i = tid; i < WF_BYTES / 16; i += TR_CHAIN) cp_async16(smem + 16 * i, a.wbf + 16 * i);
        asm volatile("cp.async.commit_group;" ::: "memory");
        const float sc = __ldcg(pdl_wait(a.scale));   // loss scale (a power of two), written by the last step's Adam kernel
        auto point = [&](int it) {
            const int s = ((int)blockIdx.x + it * (int)gridDim.x) * 128 + row;
            return a.idx ? a.idx[s] : s;
        };
        int pt = point(0);
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        handover();
        for (int it = 0; it < count; ++it) {
            // the sample's targets and the next tile's points, fetched ahead of their use
            const float* tg = a.target + (size_t)pt * a.tstride;
            float t4[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) t4[j] = half == 0 && j < a.n_out ? tg[j] : 0.f;
            if (it + 1 < count) pt = point(it + 1);
#pragma unroll 1
            for (int l = 0; l < NLAYER; ++l) {
                wait();
                // (this product came behind everything before it: the other X0 buffer has been read)
                if (l == 0 && it > 0 && it + 1 < count) bar_arrive(TB_EMPTY + ((it + 1) & 1), TR_CHAIN + TR_ENCODE);
                if (l < NLAYER - 1) {
                    float v[2][16];
                    tmem_ld16(acc + 32u * half, v[0]);
                    tmem_ld16(acc + 32u * half + 16u, v[1]);
                    tmem_wait_ld();
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        uint4 lo4, hi4;
                        relu_pack(v[h], lo4, hi4);
                        uint8_t* dst = smem + hbuf(l + 1) + kmajor_offset(row, 32 * half + 16 * h, HID);
                        *reinterpret_cast<uint4*>(dst) = lo4;
                        *reinterpret_cast<uint4*>(dst + 128) = hi4;
                    }
                    handover();
                } else {
                    // relative L2 loss (y - t)^2 / (sg(y)^2 + 0.01) and its gradient
                    float lsum = 0.f;
                    if (half == 0) {
                        float v[16];
                        tmem_ld16(acc, v);
                        tmem_wait_ld();
#pragma unroll
                        for (int j = 0; j < OUTP; ++j) {
                            float g = 0.f;
                            if (j < a.n_out) {
                                const float t = j < 4 ? t4[j & 3] : tg[j];
                                const float d = v[j] - t, den = v[j] * v[j] + 0.01f;
                                lsum += d * d / den;
                                g = 2.f * d / den * a.loss_scale * sc;
                            }
                            v[j] = g;
                        }
                        uint8_t* dst = smem + TS_DY + kmajor_offset(row, 0, OUTP);
                        *reinterpret_cast<uint4*>(dst) =
                            make_uint4(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]), pack_bf16(v[4], v[5]), pack_bf16(v[6], v[7]));
                        *reinterpret_cast<uint4*>(dst + 128) =
                            make_uint4(pack_bf16(v[8], v[9]), pack_bf16(v[10], v[11]), pack_bf16(v[12], v[13]), pack_bf16(v[14], v[15]));
                    }
                    handover();
                    if (half == 0) {
                        for (int o = 16; o > 0; o >>= 1) lsum += __shfl_xor_sync(0xffffffffu, lsum, o);
                        if (lane == 0 && ok && lsum != 0.f) atomicAdd(a.loss, lsum);
                    }
                }
            }
#pragma unroll 1
            for (int l = NLAYER - 1; l >= 1; --l) {
                const uint32_t off = kmajor_offset(row, 32 * half, HID);
                uint4 h[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) h[q] = *reinterpret_cast<const uint4*>(smem + hbuf(l) + off + 128 * q);
                wait();
                const uint32_t zn = l == 4 ? (uint32_t)TS_E : hbuf(l + 1);
                float v[2][16];
                tmem_ld16(acc + 32u * half, v[0]);
                tmem_ld16(acc + 32u * half + 16u, v[1]);
                tmem_wait_ld();
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const uint32_t hw[4] = {h[q].x, h[q].y, h[q].z, h[q].w};
                    uint32_t zw[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const __nv_bfloat162 b = *reinterpret_cast<const __nv_bfloat162*>(&hw[j]);
                        const float lo = v[q >> 1][8 * (q & 1) + 2 * j], hi = v[q >> 1][8 * (q & 1) + 2 * j + 1];
                        zw[j] = pack_bf16(__low2float(b) > 0.f ? lo : 0.f, __high2float(b) > 0.f ? hi : 0.f);
                    }
                    *reinterpret_cast<uint4*>(smem + zn + off + 128 * q) = make_uint4(zw[0], zw[1], zw[2], zw[3]);
                }
                handover();
            }
        }
        wait();   // the last dW_0
        fence_before_sync();
    }
    __syncthreads();
    fence_after_sync();
    // the CTA's weight gradients: rows = outputs 0..63, in the lanes of the warps 0 and 1 of each four
    if (warp < W_ISSUE && (warp & 3) < 2 && !gave_up) {
        const int row = (warp & 3) * 32 + lane;
        float* dw = a.dwpart + (size_t)blockIdx.x * NWEIGHT;
        int piece = 0;
        for (int l = 0; l < NLAYER; ++l) {
            const int Kin = in_dim(l), Nout = out_dim(l);
            for (int c = 0; c < Kin; c += 16, ++piece) {
                if ((piece & 3) != warp >> 2) continue;
                float v[16];
                tmem_ld16(tmem + ((uint32_t)((warp & 3) * 32) << 16) + tr_dw_col(l) + (uint32_t)c, v);
                tmem_wait_ld();
                if (row < Nout) {
                    float4* d4 = reinterpret_cast<float4*>(dw + master_off(l) + row * Kin + c);
#pragma unroll
                    for (int j = 0; j < 4; ++j) d4[j] = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
                }
            }
        }
    }
    fence_before_sync();
    __syncthreads();
    if (warp == W_ISSUE) tmem_dealloc(tmem, TR_COLS);
}

// byte offset of master weight i in the bf16 tiles
__device__ __forceinline__ uint32_t tile_offset(int i) {
    int l = 0;
    while (l + 1 < NLAYER && i >= master_off(l + 1)) ++l;
    const int K = in_dim(l), r = (i - master_off(l)) / K, k = (i - master_off(l)) % K;
    return wf_off(l) + kmajor_offset(r, k, K);
}

// Master weights (FP32, [out][in] per layer) -> bf16 tiles.
__global__ void k_mlp_pack(const float* __restrict__ w, uint8_t* __restrict__ wbf) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < NWEIGHT) st_bf16(wbf, tile_offset(i), w[i]);
}

// Loss scaling.  The output gradient is multiplied by a power-of-two scale before it goes
// through the bf16 backward pass and divided out of the summed weight gradient (exact for a power
// of two, barring overflow).  A step whose summed gradient is not finite is skipped and the
// scale halved; after SCALE_RUN finite steps in a row it doubles, up to SCALE_MAX.
// Device state, floats: scale for the next step, steps applied, finite steps in a row, steps skipped.
enum MlpState { ST_SCALE = 0, ST_STEPS, ST_RUN, ST_SKIPPED, ST_COUNT };
constexpr float SCALE_MAX = 65536.f;
constexpr int SCALE_RUN = 1000;
// Gradient of each weight = the CTAs' gradients added in a fixed order (reproducible): slice s
// of GSLICES adds CTAs s, s + GSLICES, ... in order, then the slices are added in order.  A block
// sums 64 weights, one thread per four weights and slice, all of a thread's loads in flight.
// 152 CTAs' gradients, 15 MB in the L2: 6.7 us (with the loss scale's step at its end 9 us).
constexpr int GSLICES = 16, GWEIGHTS = 64;
static_assert(NWEIGHT % GWEIGHTS == 0, "whole blocks of weights");
__global__ void __launch_bounds__(GSLICES * GWEIGHTS / 4) k_mlp_gsum(const float* __restrict__ part, int nctas, float* __restrict__ gsum,
                                                                     unsigned* __restrict__ words) {
    __shared__ float slice[GSLICES][GWEIGHTS];
    pdl_release();
    part = pdl_wait(part);
    const int w4 = threadIdx.x % (GWEIGHTS / 4), s = threadIdx.x / (GWEIGHTS / 4);
    const float4* p = reinterpret_cast<const float4*>(part) + blockIdx.x * (GWEIGHTS / 4) + w4;
    float4 g = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 5
    for (int t = s; t < nctas; t += GSLICES) {
        const float4 x = p[(size_t)t * (NWEIGHT / 4)];
        g.x += x.x;
        g.y += x.y;
        g.z += x.z;
        g.w += x.w;
    }
    *reinterpret_cast<float4*>(&slice[s][4 * w4]) = g;
    __syncthreads();
    if (threadIdx.x >= GWEIGHTS) return;
    float sum = 0.f;
#pragma unroll
    for (int k = 0; k < GSLICES; ++k) sum += slice[k][threadIdx.x];
    gsum[blockIdx.x * GWEIGHTS + threadIdx.x] = sum;
    if (!isfinite(sum)) atomicOr(words + WD_FAILED, STEP_NONFINITE);
}

// One Adam step on the FP32 master weights, and their bf16 copies; the loss scale's step.  A step of which
// a wait gave up changes nothing.  Every
// thread reads the state of before the step and forms Adam's bias corrections 1 / (1 - b^t) itself,
// in FP32 (a double pow is a long chain of the GPU's slow FP64 operations); the last block to have
// read the state writes the next one.
__global__ void __launch_bounds__(128) k_mlp_adam(const float* __restrict__ gsum, float* __restrict__ w, float* __restrict__ m1,
                                                  float* __restrict__ m2, float* __restrict__ grad, uint8_t* __restrict__ wbf, float lr, float b1,
                                                  float b2, float eps, float* st, unsigned* words) {
    const int i = blockIdx.x * 128 + threadIdx.x;
    pdl_release();
    st = pdl_wait(st);
    gsum = pdl_wait(gsum);
    words = pdl_wait(words);
    w = pdl_wait(w);
    m1 = pdl_wait(m1);
    m2 = pdl_wait(m2);
    const float4 s = __ldcg(reinterpret_cast<const float4*>(st));
    const unsigned failed = __ldcg(words + WD_FAILED);
    const bool skip = failed != 0u;
    const float scale = s.x, t = s.y + 1.f;
    if (i < NWEIGHT && !skip) {
        const float c1 = 1.f / (1.f - powf(b1, t)), c2 = 1.f / (1.f - powf(b2, t));
        const float g = gsum[i] * (1.f / scale);
        grad[i] = g;
        const float m = b1 * m1[i] + (1.f - b1) * g;
        const float v = b2 * m2[i] + (1.f - b2) * g * g;
        m1[i] = m;
        m2[i] = v;
        const float x = w[i] - lr * (m * c1) / (sqrtf(v * c2) + eps);
        w[i] = x;
        st_bf16(wbf, tile_offset(i), x);
    }
    __syncthreads();   // the block's threads have read the state
    if (threadIdx.x != 0) return;
    __threadfence();
    if (atomicAdd(words + WD_TICKET, 1u) != gridDim.x - 1) return;
    words[WD_TICKET] = 0u;
    words[WD_FAILED] = 0u;   // ready for the next step
    float4 n = s;
    if (failed & STEP_GAVE_UP) {
        // (not a matter of the scale)
    } else if (skip) {
        n.x = fmaxf(scale * 0.5f, 1.f);
        n.z = 0.f;
        n.w += 1.f;
    } else {
        n.y = t;
        n.z += 1.f;
        if (n.z >= (float)SCALE_RUN) {
            n.x = fminf(scale * 2.f, SCALE_MAX);
            n.z = 0.f;
        }
    }
    *reinterpret_cast<float4*>(st) = n;
}

}  // namespace

extern "C" rc_status rc_mlp_tile_product(const uint16_t* d_a, const uint16_t* d_b, float* d_d, int K, int N, unsigned* d_err,
                                         void* stream) {
    if (!d_a || !d_b || !d_d || !d_err || K < 16 || K > 256 || K % 16 || N < 16 || N > 256 || N % 16) return RC_ERR_ARG;
    const size_t smem = (size_t)(TILE_M + N) * K * 2;
    if (smem > 200 * 1024) return RC_ERR_ARG;
    cudaStream_t st = (cudaStream_t)stream;
    if (smem > 48 * 1024 && cudaFuncSetAttribute(k_tile_product, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
        return RC_ERR_CUDA;
    k_tile_product<<<1, 128, smem, st>>>(d_a, d_b, d_d, K, N, d_err);
    return cudaGetLastError() == cudaSuccess ? RC_OK : RC_ERR_CUDA;
}

extern "C" rc_status rc_mlp_wait_check(uint32_t polls, int arrive, unsigned* d_err, void* stream) {
    if (!d_err || polls < 1 || polls > (1u << 24)) return RC_ERR_ARG;
    k_wait_check<<<1, 32, 0, (cudaStream_t)stream>>>(polls, arrive != 0, d_err);
    return cudaGetLastError() == cudaSuccess ? RC_OK : RC_ERR_CUDA;
}

// ---------------------------------------------------------------- C ABI of the network
struct rc_mlp {
    rc_mlp_config cfg{};
    cudaStream_t stream = nullptr;
    bool own_stream = false;
    float *w = nullptr, *m1 = nullptr, *m2 = nullptr, *grad = nullptr, *part = nullptr, *gsum = nullptr, *loss = nullptr;
    float* state = nullptr;     // loss scale and Adam step state (MlpState)
    uint8_t* wbf = nullptr;
    unsigned* err = nullptr;
    unsigned* words = nullptr;  // MlpWord
    int cap_tiles = 0, sms = 0;
    uint32_t polls = WAIT_LIMIT;
    long long step = 0;
    std::string msg;
};

namespace {

rc_status mfail(rc_mlp* m, rc_status s, const char* what) {
    if (m) m->msg = what;
    return s;
}

MlpArgs args_of(const rc_mlp* m) {
    MlpArgs a{};
    a.wbf = m->wbf;
    a.n_out = m->cfg.n_out;
    for (int k = 0; k < 3; ++k) {
        a.lo[k] = m->cfg.box_lo[k];
        a.inv_ext[k] = 1.f / (m->cfg.box_hi[k] - m->cfg.box_lo[k]);
    }
    a.err = m->err;
    a.polls = m->polls;
    return a;
}

// A small counter-based generator for the initial weights (splitmix64).
uint64_t splitmix(uint64_t& s) {
    uint64_t z = (s += 0x9E3779B97F4A7C15ull);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

}  // namespace

extern "C" {

rc_status rc_mlp_create(const rc_mlp_config* cfg, rc_mlp** out) {
    if (!cfg || !out) return RC_ERR_ARG;
    *out = nullptr;
    if (cfg->n_out < 1 || cfg->n_out > OUTP || cfg->max_batch < 128 || !(cfg->lr >= 0.f)) return RC_ERR_ARG;
    for (int k = 0; k < 3; ++k)
        if (!(cfg->box_hi[k] > cfg->box_lo[k])) return RC_ERR_ARG;
    rc_mlp* m = new rc_mlp();
    m->cfg = *cfg;
    auto bad = [&](rc_status s) { rc_mlp_destroy(m); return s; };
    if (cudaSetDevice(cfg->device) != cudaSuccess) return bad(RC_ERR_CUDA);
    if (cfg->stream) m->stream = (cudaStream_t)cfg->stream;
    else {
        if (cudaStreamCreateWithFlags(&m->stream, cudaStreamNonBlocking) != cudaSuccess) return bad(RC_ERR_CUDA);
        m->own_stream = true;
    }
    cudaDeviceGetAttribute(&m->sms, cudaDevAttrMultiProcessorCount, cfg->device);
    m->cap_tiles = (cfg->max_batch + 127) / 128;
    if (cudaMalloc(&m->w, 4 * NWEIGHT) || cudaMalloc(&m->m1, 4 * NWEIGHT) || cudaMalloc(&m->m2, 4 * NWEIGHT) ||
        cudaMalloc(&m->grad, 4 * NWEIGHT) || cudaMalloc(&m->wbf, WF_BYTES) || cudaMalloc(&m->err, 4) ||
        cudaMalloc(&m->loss, 4) || cudaMalloc(&m->part, (size_t)4 * NWEIGHT * std::max(1, std::min(m->cap_tiles, m->sms))) ||
        cudaMalloc(&m->gsum, 4 * NWEIGHT) || cudaMalloc(&m->state, 4 * ST_COUNT) || cudaMalloc(&m->words, 4 * WD_COUNT))
        return bad(RC_ERR_NOMEM);
    {
        float st0[ST_COUNT] = {0};
        float sc = cfg->loss_scale > 0.f ? cfg->loss_scale : 1024.f;
        st0[ST_SCALE] = exp2f(floorf(log2f(sc)));   // a power of two
        if (cudaMemcpy(m->state, st0, sizeof st0, cudaMemcpyHostToDevice) != cudaSuccess) return bad(RC_ERR_CUDA);
    }
    // He-uniform initial weights, seeded
    std::vector<float> w(NWEIGHT);
    uint64_t st = 0x5EEDull ^ (uint64_t)cfg->seed * 0x100000001B3ull;
    for (int l = 0; l < NLAYER; ++l) {
        const float lim = sqrtf(6.f / (float)(l == 0 ? 168 : HID));
        for (int i = master_off(l); i < master_off(l) + out_dim(l) * in_dim(l); ++i) {
            const double u = (double)(splitmix(st) >> 11) * (1.0 / 9007199254740992.0);
            w[i] = (float)((2.0 * u - 1.0) * lim);
        }
        if (l == NLAYER - 1)   // unused outputs start (and stay, their gradient is zero) at zero
            for (int r = cfg->n_out; r < OUTP; ++r)
                for (int k = 0; k < HID; ++k) w[master_off(l) + r * HID + k] = 0.f;
    }
    rc_status s = rc_mlp_weights(m, w.data(), w.size(), 1);
    if (s != RC_OK) return bad(s);
    if (cudaMemsetAsync(m->m1, 0, 4 * NWEIGHT, m->stream) || cudaMemsetAsync(m->m2, 0, 4 * NWEIGHT, m->stream) ||
        cudaMemsetAsync(m->err, 0, 4, m->stream) || cudaMemsetAsync(m->words, 0, 4 * WD_COUNT, m->stream) ||
        cudaStreamSynchronize(m->stream))
        return bad(RC_ERR_CUDA);
    if (cudaFuncSetAttribute(k_mlp_train, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TRAIN_SMEM) ||
        cudaFuncSetAttribute(k_mlp_infer, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)INFER_SMEM))
        return bad(RC_ERR_CUDA);
    *out = m;
    return RC_OK;
}

void rc_mlp_destroy(rc_mlp* m) {
    if (!m) return;
    if (m->stream) cudaStreamSynchronize(m->stream);
    cudaFree(m->w); cudaFree(m->m1); cudaFree(m->m2); cudaFree(m->grad); cudaFree(m->part);
    cudaFree(m->loss); cudaFree(m->wbf); cudaFree(m->err); cudaFree(m->state); cudaFree(m->words); cudaFree(m->gsum);
    if (m->own_stream && m->stream) cudaStreamDestroy(m->stream);
    delete m;
}

const char* rc_mlp_last_error(const rc_mlp* m) { return m ? m->msg.c_str() : "no network"; }

rc_status rc_mlp_weights(rc_mlp* m, float* host, size_t n, int to_device) {
    if (!m || !host || n != (size_t)NWEIGHT) return mfail(m, RC_ERR_ARG, "weights: 24576 floats");
    if (to_device) {
        if (cudaMemcpyAsync(m->w, host, 4 * NWEIGHT, cudaMemcpyHostToDevice, m->stream) != cudaSuccess) return mfail(m, RC_ERR_CUDA, "copy");
        k_mlp_pack<<<(NWEIGHT + 255) / 256, 256, 0, m->stream>>>(m->w, m->wbf);
        if (cudaGetLastError() != cudaSuccess) return mfail(m, RC_ERR_CUDA, "pack");
    } else if (cudaMemcpyAsync(host, m->w, 4 * NWEIGHT, cudaMemcpyDeviceToHost, m->stream) != cudaSuccess) {
        return mfail(m, RC_ERR_CUDA, "copy");
    }
    return cudaStreamSynchronize(m->stream) == cudaSuccess ? RC_OK : mfail(m, RC_ERR_CUDA, "sync");
}

rc_status rc_mlp_gradients(rc_mlp* m, float* host, size_t n) {
    if (!m || !host || n != (size_t)NWEIGHT) return mfail(m, RC_ERR_ARG, "gradients: 24576 floats");
    if (cudaMemcpyAsync(host, m->grad, 4 * NWEIGHT, cudaMemcpyDeviceToHost, m->stream) != cudaSuccess ||
        cudaStreamSynchronize(m->stream) != cudaSuccess)
        return mfail(m, RC_ERR_CUDA, "copy");
    return RC_OK;
}

rc_status rc_mlp_train(rc_mlp* m, const float* d_pos4, const float* d_nrm4, const float* d_aux4, const float* d_target, int tstride,
                       const int* d_idx, int n, float* d_loss) {
    if (!m || !d_pos4 || !d_nrm4 || !d_aux4 || !d_target || n < 128 || n % 128 || n > 128 * m->cap_tiles || tstride < m->cfg.n_out)
        return mfail(m, RC_ERR_ARG, "train: n a multiple of 128 up to max_batch");
    MlpArgs a = args_of(m);
    a.P = reinterpret_cast<const float4*>(d_pos4);
    a.N = reinterpret_cast<const float4*>(d_nrm4);
    a.aux = reinterpret_cast<const float4*>(d_aux4);
    a.target = d_target;
    a.tstride = tstride;
    a.idx = d_idx;
    a.n = n;
    a.dwpart = m->part;
    a.loss = d_loss ? d_loss : m->loss;
    a.loss_scale = 1.f / ((float)n * (float)m->cfg.n_out);
    a.scale = m->state + ST_SCALE;
    a.words = m->words;
    const int ntiles = n / 128, ctas = std::min(ntiles, m->sms);
    m->step++;
    const float b1 = 0.9f, b2 = 0.99f;
    if (!d_loss && cudaMemsetAsync(m->loss, 0, 4, m->stream) != cudaSuccess) return mfail(m, RC_ERR_CUDA, "clear");
    if (launch_dependent(k_mlp_train, ctas, TR_THREADS, TRAIN_SMEM, m->stream, a, ntiles) != cudaSuccess ||
        launch_dependent(k_mlp_gsum, NWEIGHT / GWEIGHTS, GSLICES * GWEIGHTS / 4, 0, m->stream, m->part, ctas, m->gsum, m->words) != cudaSuccess ||
        launch_dependent(k_mlp_adam, NWEIGHT / 128, 128, 0, m->stream, m->gsum, m->w, m->m1, m->m2, m->grad, m->wbf, m->cfg.lr, b1, b2, 1e-8f,
                         m->state, m->words) != cudaSuccess)
        return mfail(m, RC_ERR_CUDA, "launch");
    return RC_OK;
}

rc_status rc_mlp_infer(rc_mlp* m, const float* d_pos4, const float* d_nrm4, const float* d_aux4, int n, float* d_out, int ostride) {
    if (!m || !d_pos4 || !d_nrm4 || !d_aux4 || !d_out || n < 1 || ostride < m->cfg.n_out) return mfail(m, RC_ERR_ARG, "infer");
    MlpArgs a = args_of(m);
    a.P = reinterpret_cast<const float4*>(d_pos4);
    a.N = reinterpret_cast<const float4*>(d_nrm4);
    a.aux = reinterpret_cast<const float4*>(d_aux4);
    a.n = n;
    a.out = d_out;
    a.ostride = ostride;
    const int ntiles = (n + 127) / 128;
    k_mlp_infer<<<std::min(ntiles, m->sms), IN_THREADS, INFER_SMEM, m->stream>>>(a);
    return cudaGetLastError() == cudaSuccess ? RC_OK : mfail(m, RC_ERR_CUDA, "launch");
}

rc_status rc_mlp_loss_scale(rc_mlp* m, float* scale, long long* steps, long long* skipped) {
    if (!m) return RC_ERR_ARG;
    float st[ST_COUNT];
    if (cudaMemcpyAsync(st, m->state, sizeof st, cudaMemcpyDeviceToHost, m->stream) != cudaSuccess ||
        cudaStreamSynchronize(m->stream) != cudaSuccess)
        return mfail(m, RC_ERR_CUDA, "copy");
    if (scale) *scale = st[ST_SCALE];
    if (steps) *steps = (long long)st[ST_STEPS];
    if (skipped) *skipped = (long long)st[ST_SKIPPED];
    return RC_OK;
}

rc_status rc_mlp_wait_limit(rc_mlp* m, uint32_t polls) {
    if (!m || polls > WAIT_LIMIT) return mfail(m, RC_ERR_ARG, "wait limit: at most 2^24 polls");
    m->polls = polls;
    return RC_OK;
}

rc_status rc_mlp_error_flags(rc_mlp* m, unsigned* flags) {
    if (!m || !flags) return RC_ERR_ARG;
    if (cudaMemcpyAsync(flags, m->err, 4, cudaMemcpyDeviceToHost, m->stream) != cudaSuccess ||
        cudaStreamSynchronize(m->stream) != cudaSuccess)
        return mfail(m, RC_ERR_CUDA, "copy");
    return RC_OK;
}

}  // extern "C"
