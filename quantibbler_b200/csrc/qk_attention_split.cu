// Float32 attention on tcgen05: both products on the 16-bit tensor cores, every float32 operand as a
// sum of 16-bit terms, so that the result is as exact as float32 multiply-adds.
//
// The exact attention face (attention_exact_kernel's contract, layouts and masks): q, k, v float32.  Each
// is two float16 terms, hi + lo, after scaling by a power of two (q per row, k per kv head, v per
// channel) that puts the largest magnitude at 2^14..2^15.  What the two terms leave out is at most 2^-23
// of the value, or 2^-39 of the largest one where that is more; of a product lo hi' + hi lo' + hi hi' are
// formed, the missing lo lo' is at most 2^-22 of it.  (Measured over random operands the result is nearer
// to 64 bits than float32 multiply-adds: 3.1e-7 against 4.8e-7 at 2048 keys.)  The terms of k and v are
// made once per call by two small kernels.
//
// The 2^-39 of the largest value is the one error that float32 arithmetic does not have: a large key or
// value somewhere in the sequence, seen by a row or not, costs the others bits.  So every row checks at its
// end what that can have cost it: each score at most f d 2^-9 (f: the factor from scaled scores to log2
// units; d channels of two operands of at most 2^15, off by 2^-25), each output channel at most
// (1 + 2 n / l) 2^-25 of its multiplier (v off by 2^-25; n weights of at most 2^14, off by 2^-25, on values of
// at most 2^15).  Where the first exceeds 2^-21 and 2^-21 of the row's largest score, or the second 2^-21 of the
// row's largest output, the row is marked, and attention_exact_kernel (qk_attention.cu) computes it again
// by float32 multiply-adds, as it does rows that are not finite (infinities or NaN among their operands, an
// overflow).  For normal operands both stay below that by a factor of a hundred; one entry of 10^4 among
// values of 1 is where marks begin.
//
// What bounds it: shared memory (operand reads of the tensor core and the copies' writes, 128 bytes a
// clock) and the instructions per score.  A CTA owns 128 query rows of one head; two units of four
// warps take the key blocks of 64 in turn (even, odd), each with its own running maximum, sum and
// output, merged at the end: while one unit is at its exponentials the tensor core works for the
// other, and q is in shared memory once.  A thread owns a row: no shuffles.  The weights go back to
// tensor memory as the A operand; v is read as it lies (MN-major B).
// The tensor core truncates when it adds, so sums must stay short: a block's product with v starts
// from zero, small terms first, and is added to the row's output in registers, in float32, rounded.
//
// Measured (32 / 8 heads of 128, causal, 2048 tokens): 3014 us on float32 multiply-adds, 167 us here
// (the six products alone take the tensor core about 46).
#include <cuda_fp16.h>

#include <algorithm>
#include <cmath>

#include "qk_attention_split.h"
#include "qk_tma.cuh"

namespace {

constexpr uint32_t kRows = 128, kKeys = 64;              // query rows of a CTA, keys of a block
constexpr uint32_t kTermBytes = kKeys * 128 * 2;         // one term of a k or v block, 128 channels
constexpr uint32_t kChunkBytes = kKeys * 128;            // ... 64 channels of it: 64 rows of 128 bytes
constexpr uint32_t kQChunkBytes = kRows * 128, kQTermBytes = 2 * kQChunkBytes;
constexpr uint32_t kThreads = 320, kLoadWarp = 8, kMmaWarp = 9;
constexpr uint32_t kTmemCols = 512, kUnitCols = 256, kOutCol = 128;  // unit: scores and weights, outputs
__device__ __forceinline__ constexpr uint32_t weight_col(uint32_t n) { return 64 + 32 * n; }  // of the weights' term n
constexpr float kLog2E = 1.4426950408889634f;
constexpr float kWeightScale = 16384.f;                  // weights are multiplied with v times this
constexpr float kScoreRoom = 0x1p-12f, kValueRoom = 16.f;  // 2^-21 over the 2^-9 and the 2^-25 of the bounds above
constexpr uint32_t kWaitLimit = 1u << 22;
constexpr uint32_t kMaxPeakChunks = 64;

constexpr uint32_t kTerms = 2;                           // of every operand
constexpr uint32_t kStages = 2, kStageBytes = 2 * kTerms * kTermBytes;
constexpr uint32_t kSmem = 1024 + kTerms * kQTermBytes + kStages * kStageBytes + 1024 + 512;
static_assert(kSmem <= 227 * 1024, "shared memory of a CTA");
constexpr uint32_t kSwapFloats = 2 * 64 * kRows, kStatFloats = 2 * 2 * kRows;  // the units' exchange: outputs, then m and l
static_assert(kStages * kStageBytes >= (kSwapFloats + kStatFloats) * 4, "the units' exchange lies in the ring");

struct Args {
    const float *q;
    float *out;
    uint32_t *marked;            // [batch x heads][tiles of 128 rows][4]: bits of the rows to be computed again
    const float *k_mul;          // per plane, the power of two that k's terms were divided by
    const float *v_mul;          // per plane and channel, the same of v
    size_t q_batch, q_head, q_row, o_batch, o_head, o_row;  // strides in values
    uint32_t heads, kv_heads, seq_q, seq_kv, d, dv, dpad, dvpad;
    int skew;                    // row i sees keys 0 .. i + skew (causal)
    int causal;
    float scale;                 // 1 / sqrt(d)
    int *error;
    uint32_t wait_limit;
};

__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t *v) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr), "r"(v[0]),
                 "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
                 : "memory");
}
// M = 128, N = n; float16 x float16 -> float32; b_mn: B is MN-major
__device__ __forceinline__ uint32_t instruction(uint32_t n, uint32_t b_mn) {
    return (1u << 4) | (b_mn << 16) | ((n >> 3) << 17) | ((kRows >> 4) << 24);
}
// MN-major tile in chunks of 64 channels (rows of 128 bytes, swizzled): chunks kChunkBytes apart
__device__ __forceinline__ uint64_t desc_mn(uint32_t smem_addr) {
    return umma_desc(smem_addr) | ((uint64_t)(kChunkBytes >> 4) << 16);
}
// One product of 16 contraction steps: A from shared memory / from tensor memory.
__device__ __forceinline__ void mma_ss(uint32_t d, uint64_t ad, uint64_t bd, uint32_t idesc, bool add) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}" ::"r"(d),
        "l"(ad), "l"(bd), "r"(idesc), "r"((uint32_t)add)
        : "memory");
}
__device__ __forceinline__ void mma_ts(uint32_t d, uint32_t at, uint64_t bd, uint32_t idesc, bool add) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}" ::"r"(d),
        "r"(at), "l"(bd), "r"(idesc), "r"((uint32_t)add)
        : "memory");
}
// Barrier `id` of n threads; true when all of them say so.
template <int kId, int kN>
__device__ __forceinline__ bool vote(bool ok) {
    uint32_t all;
    asm volatile(
        "{\n .reg .pred p, q;\n setp.ne.b32 p, %1, 0;\n barrier.cta.red.and.pred q, %2, %3, p;\n selp.u32 %0, 1, 0, q;\n}"
        : "=r"(all)
        : "r"((uint32_t)ok), "n"(kId), "n"(kN)
        : "memory");
    return all != 0;
}
__device__ __forceinline__ uint32_t pack_f16x2(float lo, float hi) {
    uint32_t r;
    asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
    return r;
}
__device__ __forceinline__ float2 unpack_f16x2(uint32_t u) { return __half22float2(*reinterpret_cast<__half2 *>(&u)); }
// Two values as their terms: t[0] the leading one.
__device__ __forceinline__ void split2(float a, float b, uint32_t *t) {
    t[0] = pack_f16x2(a, b);
    const float2 h = unpack_f16x2(t[0]);
    t[1] = pack_f16x2(a - h.x, b - h.y);
}
// The power of two that brings a magnitude `peak` to [2^14, 2^15), and the one that undoes it.  Peaks
// outside 2^-100 .. 2^126 (zero, infinity and NaN among them) take the nearest end of that range.
__host__ __device__ __forceinline__ int peak_exponent(uint32_t peak_bits) {
    const int e = (int)((peak_bits & 0x7fffffffu) >> 23) - 127;
    return e < -100 ? -100 : e > 126 ? 126 : e;
}
__device__ __forceinline__ float pow2(int e) { return __int_as_float((e + 127) << 23); }  // -126 <= e <= 127

// The multiplier that undoes the scaling; NaN for a plane or channel that holds an infinity or NaN (its other
// values have been scaled away), so that the rows that use it are computed by plain arithmetic; zero for zeros,
// which are exact.
__device__ __forceinline__ float undo(uint32_t peak_bits, int e) {
    return peak_bits >= 0x7f800000u ? __int_as_float(0x7fffffff) : peak_bits == 0 ? 0.f : pow2(e - 14);
}

// ------------------------------------------------------------------ terms of k and v
// Largest magnitude (as the bits of a float32) of a chunk of a plane's rows: of the whole chunk for k, per
// channel for v.  Grid (chunks, planes, k or v); a thread owns a channel, so that rows are read whole.
__global__ void __launch_bounds__(256)
kv_peaks_kernel(const float *__restrict__ k, const float *__restrict__ v, uint32_t *__restrict__ peaks, uint32_t seq,
                uint32_t d, uint32_t dv, uint32_t chunk_rows) {
    qk::pdl_launch();
    qk::pdl_wait();
    __shared__ uint32_t part[256];
    const bool is_v = blockIdx.z != 0;
    const uint32_t n = is_v ? dv : d, chunk = blockIdx.x, plane = blockIdx.y, ch = threadIdx.x % 128;
    const float *src = (is_v ? v : k) + (size_t)plane * seq * n;
    const uint32_t row1 = min(seq, (chunk + 1) * chunk_rows);
    uint32_t top = 0;
    if (ch < n)
        for (uint32_t r = chunk * chunk_rows + threadIdx.x / 128; r < row1; r += 2)
            top = max(top, __float_as_uint(src[(size_t)r * n + ch]) & 0x7fffffffu);
    part[threadIdx.x] = top;
    __syncthreads();
    // [plane][chunk][256]: v's channels, then k's partial maxima
    if (threadIdx.x < 128)
        peaks[((size_t)plane * gridDim.x + chunk) * 256 + (is_v ? 0 : 128) + threadIdx.x] =
            max(part[threadIdx.x], part[threadIdx.x + 128]);
}

// The two float16 terms of k and v, [plane][term][row][pad] (channels past the head size are zeros), and
// the multipliers that undo the scaling.  Grid (blocks of 64 rows, planes, k or v).
__global__ void __launch_bounds__(256)
kv_terms_kernel(const float *__restrict__ k, const float *__restrict__ v, const uint32_t *__restrict__ peaks,
                uint32_t n_chunks, uint32_t seq, uint32_t d, uint32_t dv, uint32_t dpad, uint32_t dvpad,
                uint16_t *__restrict__ k_terms, uint16_t *__restrict__ v_terms, float *__restrict__ k_mul,
                float *__restrict__ v_mul) {
    qk::pdl_launch();
    qk::pdl_wait();
    __shared__ uint32_t top[128];
    const bool is_v = blockIdx.z != 0;
    const uint32_t n = is_v ? dv : d, pad = is_v ? dvpad : dpad, plane = blockIdx.y;
    if (threadIdx.x < 128) {
        uint32_t t = 0;
        const uint32_t *p = peaks + (size_t)plane * n_chunks * 256 + (is_v ? 0 : 128) + threadIdx.x;
        for (uint32_t c = 0; c < n_chunks; ++c) t = max(t, p[c * 256]);
        top[threadIdx.x] = t;
    }
    __syncthreads();
    if (!is_v)  // one scale for the head
        for (int off = 64; off > 0; off >>= 1) {
            if (threadIdx.x < off) top[threadIdx.x] = max(top[threadIdx.x], top[threadIdx.x + off]);
            __syncthreads();
        }
    const uint32_t pairs = pad / 2, pr = threadIdx.x % pairs, c = 2 * pr;
    const int e0 = peak_exponent(top[is_v ? c : 0]), e1 = peak_exponent(top[is_v ? c + 1 : 0]);
    if (blockIdx.x == 0 && threadIdx.x < pairs) {
        if (is_v) {
            v_mul[(size_t)plane * dvpad + c] = undo(top[c], e0);
            v_mul[(size_t)plane * dvpad + c + 1] = undo(top[c + 1], e1);
        } else if (pr == 0) {
            k_mul[plane] = undo(top[0], e0);
        }
    }
    const float m0 = pow2(14 - e0), m1 = pow2(14 - e1);
    const float *src = (is_v ? v : k) + (size_t)plane * seq * n;
    uint16_t *dst = (is_v ? v_terms : k_terms) + (size_t)plane * 2 * seq * pad;
    const uint32_t row1 = min(seq, (blockIdx.x + 1) * kKeys);
    for (uint32_t r = blockIdx.x * kKeys + threadIdx.x / pairs; r < row1; r += 256 / pairs) {
        const float a = c < n ? src[(size_t)r * n + c] * m0 : 0.f, b = c + 1 < n ? src[(size_t)r * n + c + 1] * m1 : 0.f;
        uint32_t t[2];
        split2(a, b, t);
        *reinterpret_cast<uint32_t *>(dst + (size_t)r * pad + c) = t[0];
        *reinterpret_cast<uint32_t *>(dst + ((size_t)seq + r) * pad + c) = t[1];
    }
}

// ------------------------------------------------------------------ the kernel
template <uint32_t kChunks>  // kChunks: head size in chunks of 64 channels (padded)
__global__ void __launch_bounds__(kThreads, 1)
split_attention_kernel(const __grid_constant__ CUtensorMap k_map, const __grid_constant__ CUtensorMap v_map, Args a) {
    qk::pdl_launch();
    extern __shared__ __align__(1024) uint8_t raw_smem[];
    uint8_t *qs = reinterpret_cast<uint8_t *>(((uintptr_t)raw_smem + 1023) & ~(uintptr_t)1023);
    uint8_t *ring = qs + kTerms * kQTermBytes;
    float *row_peak = reinterpret_cast<float *>(ring + kStages * kStageBytes);  // [2][128]
    uint64_t *q_full = reinterpret_cast<uint64_t *>(row_peak + 256);
    uint64_t *k_full = q_full + 1, *k_empty = k_full + kStages, *v_full = k_empty + kStages, *v_empty = v_full + kStages;
    uint64_t *s_full = v_empty + kStages, *p_full = s_full + 2, *o_full = p_full + 2, *drain = o_full + 2;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(drain + 1);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
    volatile int *never = reinterpret_cast<volatile int *>(tmem_slot + 2);
    uint32_t *marks = tmem_slot + 3;  // [4] rows to be computed again
    const uint32_t warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    const uint32_t head = blockIdx.x % a.heads, batch = blockIdx.x / a.heads, kvh = head / (a.heads / a.kv_heads);
    const uint32_t plane = batch * a.kv_heads + kvh;
    const uint32_t row0 = (gridDim.y - 1 - blockIdx.y) * kRows;   // (late rows see most keys: they go first)
    const uint32_t rows = min(kRows, a.seq_q - row0);
    const uint32_t n_keys = a.causal ? min(a.seq_kv, (uint32_t)((int)(row0 + rows) + a.skew)) : a.seq_kv;
    const uint32_t n_blocks = (n_keys + kKeys - 1) / kKeys;
    const uint32_t d_chunks = kChunks, v_chunks = a.dvpad / 64;
    if (threadIdx.x == 0) {
        mbar_init(q_full, 8);
        for (uint32_t s = 0; s < kStages; ++s) {
            mbar_init(k_full + s, 1);
            mbar_init(k_empty + s, 1);
            mbar_init(v_full + s, 1);
            mbar_init(v_empty + s, 1);
        }
        for (int u = 0; u < 2; ++u) {
            mbar_init(s_full + u, 1);
            mbar_init(p_full + u, 4);
            mbar_init(o_full + u, 1);
        }
        mbar_init(drain, 1);
        *abort_flag = 0;
        *never = 0;
        for (int i = 0; i < 4; ++i) marks[i] = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&k_map) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&v_map) : "memory");
    }
    if (warp == kMmaWarp) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(kTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    qk::pdl_wait();
    const uint32_t tmem = *tmem_slot;
    uint32_t fetched_k = 0, fetched_v = 0;  // (loading warp) blocks whose copies have been issued

    if (warp == kLoadWarp) {
        for (uint32_t g = 0; g < n_blocks; ++g) {
            const uint32_t s = g % kStages, parity = ((g / kStages) & 1) ^ 1;
            uint8_t *stage = ring + s * kStageBytes;
            if (!mbar_wait(k_empty + s, parity, abort_flag, a.wait_limit)) {
                *abort_flag = 1;
                break;
            }
            if (lane == 0) {
                mbar_expect(k_full + s, kTerms * d_chunks * kChunkBytes);
                for (uint32_t t = 0; t < kTerms; ++t)
                    for (uint32_t c = 0; c < d_chunks; ++c)
                        tma_load_3d(smem_u32(stage + t * kTermBytes + c * kChunkBytes), &k_map, c * 64, g * kKeys,
                                    plane * kTerms + t, k_full + s);
            }
            fetched_k = g + 1;
            __syncwarp();
            if (!mbar_wait(v_empty + s, parity, abort_flag, a.wait_limit)) {
                *abort_flag = 1;
                break;
            }
            if (lane == 0) {
                mbar_expect(v_full + s, kTerms * v_chunks * kChunkBytes);
                for (uint32_t t = 0; t < kTerms; ++t)
                    for (uint32_t c = 0; c < v_chunks; ++c)
                        tma_load_3d(smem_u32(stage + (kTerms + t) * kTermBytes + c * kChunkBytes), &v_map, c * 64,
                                    g * kKeys, plane * kTerms + t, v_full + s);
            }
            fetched_v = g + 1;
            __syncwarp();
        }
    } else if (warp == kMmaWarp) {
        const uint32_t idesc_s = instruction(kKeys, 0), idesc_o = instruction(a.dvpad, 1);
        // (descriptors differ in their address field alone: sixteen bytes a unit)
        const uint64_t q_desc = umma_desc(smem_u32(qs)), k_desc = umma_desc(smem_u32(ring));
        const uint64_t v_desc = desc_mn(smem_u32(ring) + kTerms * kTermBytes);
        // scores of block g into its unit's columns: small terms first
        auto scores = [&](uint32_t g) {  // (one lane)
            const uint64_t kd = k_desc + (uint64_t)((g % kStages) * (kStageBytes >> 4));
            const uint32_t dst = tmem + kUnitCols * (g & 1);
#pragma unroll
            for (uint32_t i = 0; i < 3; ++i) {
                const uint32_t tq = i == 0 ? 1 : 0, tk = i == 1 ? 1 : 0;
#pragma unroll
                for (uint32_t k = 0; k < 4 * kChunks; ++k)
                    mma_ss(dst, q_desc + ((tq * kQTermBytes + k / 4 * kQChunkBytes + k % 4 * 32) >> 4),
                           kd + ((tk * kTermBytes + k / 4 * kChunkBytes + k % 4 * 32) >> 4), idesc_s, i + k != 0);
            }
            umma_commit(k_empty + g % kStages);
            umma_commit(s_full + (g & 1));
        };
        auto values = [&](uint32_t g) {  // (one lane)
            const uint64_t vd = v_desc + (uint64_t)((g % kStages) * (kStageBytes >> 4));
            const uint32_t unit = tmem + kUnitCols * (g & 1);
#pragma unroll
            for (uint32_t i = 0; i < 3; ++i) {
                const uint32_t tp = i == 0 ? 1 : 0, tv = i == 1 ? 1 : 0;
#pragma unroll
                for (uint32_t k = 0; k < kKeys / 16; ++k)
                    mma_ts(unit + kOutCol, unit + weight_col(tp) + k * 8, vd + ((tv * kTermBytes + k * 2048) >> 4), idesc_o,
                           i + k != 0);
            }
            umma_commit(v_empty + g % kStages);
            umma_commit(o_full + (g & 1));
        };
        bool ok = mbar_wait(q_full, 0, abort_flag, a.wait_limit);
        for (uint32_t g = 0; g < 2 && g < n_blocks && ok; ++g) {
            ok = mbar_wait(k_full + g % kStages, 0, abort_flag, a.wait_limit);
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (elect_one()) scores(g);
            __syncwarp();
        }
        for (uint32_t g = 0; g < n_blocks && ok; ++g) {
            ok = mbar_wait(v_full + g % kStages, (g / kStages) & 1, abort_flag, a.wait_limit);
            if (ok) ok = mbar_wait(p_full + (g & 1), (g >> 1) & 1, abort_flag, a.wait_limit);
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (elect_one()) values(g);
            __syncwarp();
            if (g + 2 >= n_blocks) continue;
            ok = mbar_wait(k_full + (g + 2) % kStages, ((g + 2) / kStages) & 1, abort_flag, a.wait_limit);
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (elect_one()) scores(g + 2);   // (over scores that the unit has read: it has handed in their weights)
            __syncwarp();
        }
        if (!ok) *abort_flag = 1;
    } else {
        const uint32_t u = warp / 4, r = threadIdx.x % 128;
        const uint32_t i = row0 + r;                      // query row
        const float *q_row = a.q + batch * a.q_batch + head * a.q_head + (size_t)min(i, a.seq_q - 1) * a.q_row;
        // q: a unit takes one chunk of 64 channels; thread = row
        float f = a.scale * kLog2E;                       // what turns a raw score into log2 units
        {
            const bool live = r < rows && u < d_chunks;
            float x[64];
            const bool wide = (a.d & 3) == 0 && (a.q_row & 3) == 0 && ((uintptr_t)q_row & 15) == 0;
#pragma unroll
            for (int c = 0; c < 64; c += 4) {
                const uint32_t ch = u * 64 + c;
                if (live && wide && ch + 4 <= a.d) {
                    const float4 t = *reinterpret_cast<const float4 *>(q_row + ch);
                    x[c] = t.x, x[c + 1] = t.y, x[c + 2] = t.z, x[c + 3] = t.w;
                } else {
#pragma unroll
                    for (int e = 0; e < 4; ++e) x[c + e] = live && ch + e < a.d ? q_row[ch + e] : 0.f;
                }
            }
            uint32_t top = 0;
#pragma unroll
            for (int c = 0; c < 64; ++c) top = max(top, __float_as_uint(x[c]) & 0x7fffffffu);
            row_peak[u * 128 + r] = __uint_as_float(top);
            asm volatile("bar.sync 3, 256;" ::: "memory");
            const int e = peak_exponent(max(top, __float_as_uint(row_peak[(u ^ 1) * 128 + r])));
            const float mul = pow2(14 - e);
            f = f * pow2(e - 14) * a.k_mul[plane];
            if (u < d_chunks) {
#pragma unroll
                for (int c = 0; c < 8; ++c) {
                    uint32_t t[4][kTerms];
#pragma unroll
                    for (int e = 0; e < 4; ++e) split2(x[8 * c + 2 * e] * mul, x[8 * c + 2 * e + 1] * mul, t[e]);
#pragma unroll
                    for (int n = 0; n < (int)kTerms; ++n)
                        *reinterpret_cast<uint4 *>(qs + n * kQTermBytes + u * kQChunkBytes + r * 128 + ((c ^ (r & 7)) << 4)) =
                            make_uint4(t[0][n], t[1][n], t[2][n], t[3][n]);
                }
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(q_full);
        }
        const uint32_t unit = tmem + kUnitCols * u + (((warp % 4) * 32) << 16);
        // keys that this row sees
        const int seen = a.causal ? min((int)i + a.skew + 1, (int)a.seq_kv) : (int)a.seq_kv;
        const int seen0 = a.causal ? min((int)row0 + a.skew + 1, (int)a.seq_kv) : (int)a.seq_kv;  // ... its tile's first row
        float m = -INFINITY, l = 0.f;
        float o[128];
#pragma unroll
        for (int c = 0; c < 128; ++c) o[c] = 0.f;
        bool ok = true;
        for (uint32_t g = u, it = 0; g < n_blocks; g += 2, ++it) {
            const int key0 = (int)(g * kKeys);
            ok = u ? vote<2, 128>(mbar_wait(s_full + 1, it & 1, abort_flag, a.wait_limit))
                   : vote<1, 128>(mbar_wait(s_full, it & 1, abort_flag, a.wait_limit));
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const bool edge = key0 + (int)kKeys > seen0;  // some row of the tile does not see the whole block
            const int limit = seen - key0;                // keys of the block that this row sees
            float top = -INFINITY;
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                uint32_t s[32];
                tmem_ld32(unit + 32 * half, s);
                tmem_ld_wait();
                float t4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
                if (edge) {
#pragma unroll
                    for (int e = 0; e < 32; ++e)
                        t4[e % 4] = fmaxf(t4[e % 4], 32 * half + e < limit ? __uint_as_float(s[e]) : -INFINITY);
                } else {
#pragma unroll
                    for (int e = 0; e < 32; ++e) t4[e % 4] = fmaxf(t4[e % 4], __uint_as_float(s[e]));
                }
                top = fmaxf(top, fmaxf(fmaxf(t4[0], t4[1]), fmaxf(t4[2], t4[3])));
            }
            const float m_new = fmaxf(m, top * f);
            const float base = m_new == -INFINITY ? 0.f : m_new;  // (nothing seen yet: every weight is zero)
            const float alpha = ex2(m - base);
            m = m_new;
            const float2 f2 = make_float2(f, f), base2 = make_float2(-base, -base);
            float2 sum = make_float2(0.f, 0.f);
#pragma unroll
            for (int part = 0; part < 4; ++part) {
                uint32_t s[16], t[kTerms][8];
                tmem_ld16(unit + 16 * part, s);
                tmem_ld_wait();
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    float2 x = __ffma2_rn(make_float2(__uint_as_float(s[2 * e]), __uint_as_float(s[2 * e + 1])), f2, base2);
                    if (edge) {
                        x.x = 16 * part + 2 * e < limit ? x.x : -INFINITY;
                        x.y = 16 * part + 2 * e + 1 < limit ? x.y : -INFINITY;
                    }
                    x = make_float2(ex2(x.x), ex2(x.y));
                    sum = __fadd2_rn(sum, x);
                    // (times 2^14 afterwards: added to the exponent's argument it would cost four bits of it)
                    x = __fmul2_rn(x, make_float2(kWeightScale, kWeightScale));
                    uint32_t w[kTerms];
                    split2(x.x, x.y, w);
#pragma unroll
                    for (int n = 0; n < (int)kTerms; ++n) t[n][e] = w[n];
                }
#pragma unroll
                for (int n = 0; n < (int)kTerms; ++n) tmem_st8(unit + weight_col(n) + 8 * part, t[n]);
            }
            l = fmaf(l, alpha, sum.x + sum.y);
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(p_full + u);
            // the block's product joins the output (in registers: the sum is rounded, not truncated)
            ok = u ? vote<2, 128>(mbar_wait(o_full + 1, it & 1, abort_flag, a.wait_limit))
                   : vote<1, 128>(mbar_wait(o_full, it & 1, abort_flag, a.wait_limit));
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
            for (int part = 0; part < 4; ++part) {
                if (part * 32 >= (int)a.dvpad) break;
                uint32_t w[32];
                tmem_ld32(unit + kOutCol + 32 * part, w);
                tmem_ld_wait();
#pragma unroll
                for (int c = 0; c < 32; c += 2) {
                    const float2 x = __ffma2_rn(make_float2(o[32 * part + c], o[32 * part + c + 1]), make_float2(alpha, alpha),
                                                make_float2(__uint_as_float(w[c]), __uint_as_float(w[c + 1])));
                    o[32 * part + c] = x.x, o[32 * part + c + 1] = x.y;
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        }
        if (!ok) *abort_flag = 1;
        // The units merge: each finishes 64 channels and hands the other 64 over, through the ring (every
        // product has been read out, every copy consumed once both units are here).
        ok = vote<3, 256>(ok);
        if (ok) {
            float *swap = reinterpret_cast<float *>(ring), *stat = swap + kSwapFloats;  // [unit][64][128], [unit][m, l][128]
            float *mine = swap + u * 64 * 128;
#pragma unroll
            for (int c = 0; c < 64; ++c) mine[c * 128 + r] = u ? o[c] : o[64 + c];
            stat[u * 256 + r] = m;
            stat[u * 256 + 128 + r] = l;
            asm volatile("bar.sync 3, 256;" ::: "memory");
            const float m2 = stat[(u ^ 1) * 256 + r], l2 = stat[(u ^ 1) * 256 + 128 + r];
            const float top = fmaxf(m, m2), base = top == -INFINITY ? 0.f : top;
            const float w1 = ex2(m - base), w2 = ex2(m2 - base);
            const float sum = l * w1 + l2 * w2, inv = 1.0f / sum, a1 = w1 * inv, a2 = w2 * inv;
            const float *other = swap + (u ^ 1) * 64 * 128;
            const float *v_mul = a.v_mul + (size_t)plane * a.dvpad;
            float *dst = a.out + batch * a.o_batch + head * a.o_head + (size_t)min(i, a.seq_q - 1) * a.o_row;
            const bool wide = (a.dv & 3) == 0 && (a.o_row & 3) == 0 && ((uintptr_t)dst & 15) == 0;
            float largest = 0.f, v_unit = 0.f;   // this unit's largest output and multiplier
            bool mark = !(f * (float)a.d <= kScoreRoom * fmaxf(1.f, fabsf(top)));
#pragma unroll
            for (int c = 0; c < 64; c += 4) {
                const uint32_t ch = u * 64 + c;
                if (r >= rows || ch >= a.dv) continue;
                float x[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const float own = u ? o[64 + c + e] : o[c + e];
                    x[e] = fmaf(own, a1, other[(c + e) * 128 + r] * a2);
                    x[e] *= v_mul[ch + e] * (1.f / kWeightScale);
                    mark = mark || !(fabsf(x[e]) < INFINITY);
                    largest = fmaxf(largest, fabsf(x[e]));
                    v_unit = fmaxf(v_unit, v_mul[ch + e]);
                }
                if (wide) {
                    *reinterpret_cast<float4 *>(dst + ch) = make_float4(x[0], x[1], x[2], x[3]);
                } else {
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        if (ch + e < a.dv) dst[ch + e] = x[e];
                }
            }
            row_peak[u * 128 + r] = largest;
            asm volatile("bar.sync 3, 256;" ::: "memory");
            largest = fmaxf(largest, row_peak[(u ^ 1) * 128 + r]);
            mark = mark || !((1.f + 2.f * (float)seen / sum) * v_unit <= kValueRoom * largest);
            const uint32_t bits = __ballot_sync(0xffffffffu, mark && r < rows);
            if (lane == 0 && bits) atomicOr(marks + warp % 4, bits);
            asm volatile("bar.sync 3, 256;" ::: "memory");
            if (threadIdx.x < 4) a.marked[((size_t)blockIdx.x * gridDim.y + row0 / kRows) * 4 + threadIdx.x] = marks[threadIdx.x];
        }
    }
    __syncwarp();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == kLoadWarp && *abort_flag) {  // the copies still in flight
        for (uint32_t g = fetched_k > kStages ? fetched_k - kStages : 0; g < fetched_k; ++g)
            (void)mbar_wait(k_full + g % kStages, (g / kStages) & 1, never, kWaitLimit);
        for (uint32_t g = fetched_v > kStages ? fetched_v - kStages : 0; g < fetched_v; ++g)
            (void)mbar_wait(v_full + g % kStages, (g / kStages) & 1, never, kWaitLimit);
    }
    if (warp == kMmaWarp && *abort_flag) {  // the products still in flight (whichever warp gave up)
        if (elect_one()) umma_commit(drain);
        __syncwarp();
        (void)mbar_wait(drain, 0, never, kWaitLimit);
    }
    if (warp == kMmaWarp)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
    if (threadIdx.x == 0 && *abort_flag) atomicOr(a.error, 1);
}

// A plane of rows of `pad` 16-bit values, `seq` of them live, planes `plane_bytes` apart.
qk_status plane_map(const void *base, size_t pad, size_t seq, size_t planes, size_t plane_bytes, CUtensorMap *out) {
    const cuuint64_t dims[3] = {pad, seq, planes};
    const cuuint64_t strides[2] = {pad * 2, plane_bytes};
    const cuuint32_t box[3] = {64, kKeys, 1};
    return encode_bf16_map(base, 3, dims, strides, box, out);
}

qk_status launch_split(qk_ctx *c, const CUtensorMap &km, const CUtensorMap &vm, Args &a, size_t batch) {
    a.error = (int *)c->d_err.ptr;
    a.wait_limit = c->wait_limit ? c->wait_limit : kWaitLimit;
    auto kernel = a.dpad == 64 ? split_attention_kernel<1> : split_attention_kernel<2>;
    QK_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem));
    const dim3 grid((unsigned)(batch * a.heads), (unsigned)qk::ceil_div(a.seq_q, kRows));
    (void)qk::launch_pdl(c->pdl, kernel, grid, dim3(kThreads), (size_t)kSmem, c->stream, km, vm, a);
    QK_CUDA(cudaGetLastError());
    c->launches++;
    c->err_armed = true;
    return QK_OK;
}

}  // namespace

namespace qk {

bool attention_split_takes(qk_ctx *c, const qk_attention_shape *s, int causal) {
    if (s->head_dim > 128 || s->val_dim > 128 || (causal && s->seq_q > s->seq_kv)) return false;
    // Below 192 keys the float32 kernel is the more exact one (error against 64 bits at 128 keys 1.7e-7 to
    // 2.5e-7 there, 1.8e-7 to 2.6e-7 here; from 192 on equal, at 2048 4.8e-7 and 3.1e-7).
    if (s->seq_kv < 192) return false;
    // Heads of up to 16 channels are padded to 64 here and cost the float32 kernel a quarter of what 64 do: up to 255
    // keys they stay there (16 channels, 32 heads: 192 tokens 16.5 against 17.9 us, one query row on 192 keys in a batch
    // of four 14.4 against 21.7; 256 tokens 22.6 against 18.1).  So do one to three value channels, where an output
    // near zero marks its row (one channel, 32 heads, 384 tokens: 43 against 48 us).
    if ((std::max(s->head_dim, s->val_dim) <= 16 && s->seq_kv < 256) || s->val_dim < 4) return false;
    if (ceil_div(s->seq_q, kRows) > 65535 || s->batch * s->n_kv_heads > 65535 || s->seq_kv > (1u << 30)) return false;
    // (a captured graph may be replayed after the scratch has moved: a recording keeps the plain kernel)
    return !capturing(c);
}

qk_status attention_split_exact(qk_ctx *c, const float *q, const float *k, const float *v, float *out,
                                const qk_attention_shape *s, int causal, const uint32_t **marked) {
    const size_t planes = s->batch * s->n_kv_heads, seq = s->seq_kv;
    const size_t dpad = s->head_dim <= 64 ? 64 : 128, dvpad = s->val_dim <= 64 ? 64 : 128;
    const size_t chunk_rows = std::max<size_t>(kKeys, ceil_div(seq, kMaxPeakChunks)), chunks = ceil_div(seq, chunk_rows);
    auto up = [](size_t n) { return (n + 255) / 256 * 256; };
    const size_t k_bytes = up(planes * 2 * seq * dpad * 2), v_bytes = up(planes * 2 * seq * dvpad * 2);
    const size_t peak_bytes = up(planes * chunks * 256 * 4), kmul_bytes = up(planes * 4);
    const size_t vmul_bytes = up(planes * dvpad * 4), mark_bytes = s->batch * s->n_heads * ceil_div(s->seq_q, kRows) * 16;
    qk_status st = error_word(c);
    if (st != QK_OK) return st;
    st = c->d_terms.reserve(k_bytes + v_bytes + peak_bytes + kmul_bytes + vmul_bytes + mark_bytes);
    if (st != QK_OK) return st;
    uint8_t *base = (uint8_t *)c->d_terms.ptr;
    uint16_t *kt = (uint16_t *)base, *vt = (uint16_t *)(base + k_bytes);
    uint32_t *peaks = (uint32_t *)(base + k_bytes + v_bytes);
    float *k_mul = (float *)(base + k_bytes + v_bytes + peak_bytes), *v_mul = (float *)((uint8_t *)k_mul + kmul_bytes);
    (void)launch_pdl(c->pdl, kv_peaks_kernel, dim3((unsigned)chunks, (unsigned)planes, 2), dim3(256), 0, c->stream, k, v, peaks,
                     (uint32_t)seq, (uint32_t)s->head_dim, (uint32_t)s->val_dim, (uint32_t)chunk_rows);
    QK_CUDA(cudaGetLastError());
    (void)launch_pdl(c->pdl, kv_terms_kernel, dim3((unsigned)ceil_div(seq, kKeys), (unsigned)planes, 2), dim3(256), 0, c->stream,
                     k, v, (const uint32_t *)peaks, (uint32_t)chunks, (uint32_t)seq, (uint32_t)s->head_dim,
                     (uint32_t)s->val_dim, (uint32_t)dpad, (uint32_t)dvpad, kt, vt, k_mul, v_mul);
    QK_CUDA(cudaGetLastError());
    c->launches += 2;
    CUtensorMap km, vm;
    if ((st = plane_map(kt, dpad, seq, planes * 2, seq * dpad * 2, &km)) != QK_OK) return st;
    if ((st = plane_map(vt, dvpad, seq, planes * 2, seq * dvpad * 2, &vm)) != QK_OK) return st;
    Args a{};
    a.q = q, a.out = out;
    a.marked = (uint32_t *)((uint8_t *)v_mul + vmul_bytes);
    a.k_mul = k_mul, a.v_mul = v_mul;
    a.q_row = s->head_dim, a.q_head = s->seq_q * s->head_dim, a.q_batch = s->n_heads * a.q_head;
    a.o_row = s->val_dim, a.o_head = s->seq_q * s->val_dim, a.o_batch = s->n_heads * a.o_head;
    a.heads = (uint32_t)s->n_heads, a.kv_heads = (uint32_t)s->n_kv_heads;
    a.seq_q = (uint32_t)s->seq_q, a.seq_kv = (uint32_t)seq;
    a.d = (uint32_t)s->head_dim, a.dv = (uint32_t)s->val_dim, a.dpad = (uint32_t)dpad, a.dvpad = (uint32_t)dvpad;
    a.skew = (int)seq - (int)s->seq_q, a.causal = causal != 0;
    a.scale = 1.0f / sqrtf((float)s->head_dim);
    if ((st = launch_split(c, km, vm, a, s->batch)) != QK_OK) return st;
    *marked = a.marked;
    return QK_OK;
}

}  // namespace qk
