// The few-instance GEMV stage by sums: what qk_gemv.cu launches where a stage of one or a few layers is too
// small to fill the machine (one token through one linear, a decode step at batch 1).
//
// Such a stage is a chain of latencies, and in the bit-sliced form its longest link is the digit table, about 150
// instructions an entry in every block.  Here there is no table.  An entry is put on the same fixed-point grid,
// v ~ q * 2^-shift with |q| < 2^47, and split in two: q = hi * 2^21 + lo.  A thread adds up hi and lo over its sixteen
// entries under the weight bits (sum_k s_k q_k = 2 * sum_{bit_k = 1} q_k - sum_k q_k), a row's sums go on as 64-bit
// integers: the same whole number as in the bit-sliced form, hence the same bits of the result.  Measured on B200, cycles
// a warp and weight on one scheduler: one 32-bit addition under a predicate 2.0, two 2.9 (a float64 one 5.3).  Under
// bfloat16 serving the lo of a warp's entries are nearly always all zero (eight bits, within 2^18 of the largest): one
// addition.
//
// A block of 512 threads owns `rows_per_block` rows.  A thread owns sixteen consecutive entries of the vector, in
// registers, and adds them up for its rows; `lanes` threads (whole warps) cover the vector, and the block's 16 warps
// make as many groups of rows as fit.  Loops are kept rolled: a launch runs most of this once, and code that has to be
// fetched costs more than a branch.  The weight rows are copied to shared memory before the wait for the kernel
// before this one.  An SM holds one block (the launch asks for that much shared memory): blocks that came in early
// beside the kernel before would crowd on some SMs and leave others idle.  Long vectors are split over the CTAs of a
// cluster, `slice_bits` entries each, on one grid, that of the whole vector's largest entry; the CTAs share out the rows, whose
// whole numbers they add up before they are converted.
//
// What bounds it: latencies.  By the clock of block 0, us from the wait to the end: the first stage of a 4096 x 4096 linear of
// rank 1102 with the norm inside 5.3 (entries 1.7, grid and conversion 0.9, sums 1.7, rows 0.8), its second stage 2.9; a
// boundary between kernels 1.1.  One 4096 x 4096 linear of rank 1024 on one token 13.4 -> 8.0 us, an eight-block step of
// width 4096 at batch 1 901 -> 731 us when it came in.  Issue slots 40 % busy while a block is there.
#pragma once

namespace {

constexpr int kSumThreads = 512, kSumEntries = 16;  // entries a thread
constexpr uint32_t kSumSlice = kSumThreads * kSumEntries;  // most entries of a CTA
constexpr int kSumLow = 21;                          // bits of lo
constexpr uint32_t kSumRanks = 8;                    // most CTAs of a cluster
// |q| <= 2^47: a row's sum over fewer entries than this is a 64-bit integer.
constexpr uint32_t kSumMostEntries = (1u << 16) - 1;

// Shared memory: [hi of the entries, transposed][lo][the entries][weight rows][partial sums][row sums]
struct SumLayout {
    uint32_t lanes, warps;  // threads over the vector (a multiple of 32), and in warps
    uint32_t pitch;         // bytes of a weight row's slice
    uint32_t low, entries, slab, part, row_sum, bytes;
};
__host__ __device__ inline SumLayout sum_layout(uint32_t slice, uint32_t rows, uint32_t entry_bytes) {
    SumLayout l;
    l.lanes = (slice + 32 * kSumEntries - 1) / (32 * kSumEntries) * 32;
    l.warps = l.lanes / 32;
    l.pitch = (slice + 127) / 128 * 16;
    l.low = kSumEntries * (l.lanes + 1) * 4;
    l.entries = 2 * l.low;
    l.slab = (l.entries + kSumEntries * l.lanes * entry_bytes + 15) / 16 * 16;
    // (a thread past the end of the slice reads past its row; its entries are zero)
    l.part = l.slab + (rows * l.pitch + l.lanes * kSumEntries / 8 + 15) / 16 * 16;
    l.row_sum = l.part + (rows + 1) * l.warps * 8;
    l.bytes = l.row_sum + rows * 8;
    return l;
}
__device__ __forceinline__ float round_bf16_fast(float v) {  // (a NaN becomes another NaN)
    uint16_t h;
    asm("cvt.rn.bf16.f32 %0, %1;" : "=h"(h) : "f"(v));
    return __uint_as_float((uint32_t)h << 16);
}

template <bool kRoundBf16, bool kFinal>
__device__ __forceinline__ void sum_form(const StageParams &p, uint32_t rows_per_block, uint32_t slice_bits, uint32_t rank,
                                         uint32_t n_rank) {
    // (aligned as everywhere in this file: the declarations are one symbol, and the first one decides for all of them; with 16
    // the streaming kernels' digit tables began half a line off, 163 -> 165 us for a stack of layers)
    extern __shared__ __align__(128) uint8_t smem_dyn[];
    // (the second stage's input is the float64 intermediate; rounded to bfloat16 it is a float32 too)
    using Entry = typename std::conditional<kFinal && !kRoundBf16, double, float>::type;
    using Bits = typename std::conditional<sizeof(Entry) == 8, unsigned long long, uint32_t>::type;
    constexpr int kWarps = kSumThreads / 32;
    __shared__ __align__(16) float norm_red[kWarps];
    __shared__ Bits top_red[kWarps];
    __shared__ Bits peer_top[kSumRanks];  // (slices)
    const uint32_t tid = threadIdx.x, warp = tid / 32, lane = tid % 32;
    const uint32_t n_rows = p.n_rows, n_bits = p.n_bits;
    const uint32_t row0 = (blockIdx.x / n_rank) * rows_per_block;
    // (an instance with fewer rows, or fewer slices, than the launch's widest; all CTAs of a cluster alike)
    if (row0 >= n_rows) {
        qk::pdl_wait();
        return;
    }
    if (n_rank > 1) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");  // (this CTA has begun)
    const uint32_t rows = min(rows_per_block, n_rows - row0);
    const uint32_t k_lo = min(rank * slice_bits, n_bits), k_hi = min(k_lo + slice_bits, n_bits);
    const SumLayout lay = sum_layout(max(1u, k_hi - k_lo), rows_per_block, sizeof(Entry));
    int *zh = reinterpret_cast<int *>(smem_dyn);  // entry k of the slice at [k % 16][k / 16], rows of lanes + 1
    int *zl = reinterpret_cast<int *>(smem_dyn + lay.low);
    Entry *entries = reinterpret_cast<Entry *>(smem_dyn + lay.entries);
    uint8_t *slab = smem_dyn + lay.slab;
    // [row][warp of the vector]; row `rows_per_block`: totals
    long long *part = reinterpret_cast<long long *>(smem_dyn + lay.part);
    long long *row_sum = reinterpret_cast<long long *>(smem_dyn + lay.row_sum);  // (slices)
    const uint32_t z_pitch = lay.lanes + 1, padded = kSumEntries * lay.lanes;

    // ---- what depends on no other kernel: the weight rows, the constant vectors
    {
        const uint32_t pieces = lay.pitch / 16, stride = (n_bits + 127) / 128 * 16;
        const uint8_t *src = p.w_rows + (size_t)row0 * stride + k_lo / 8;
        if (k_hi > k_lo)
#pragma unroll 1
            for (uint32_t i = tid; i < rows * pieces; i += kSumThreads) {
                const uint32_t r = i / pieces, piece = i - r * pieces;
                cp_async16(slab + r * lay.pitch + piece * 16, src + (size_t)r * stride + piece * 16);
            }
        cp_async_commit();
        if (!kFinal && p.in_scale && !p.norm_w && tid * 32 < k_hi - k_lo)  // (a line a thread: the slice is at most 8192)
            asm volatile("prefetch.global.L2 [%0];" ::"l"(p.in_scale + k_lo + tid * 32));
    }
    const uint32_t my_row = min(row0 + tid, n_rows - 1);
    const float row_scale = kFinal && p.out_scale ? __ldg(p.out_scale + my_row) : 1.f;
    const float row_bias = kFinal && p.out_bias ? __ldg(p.out_bias + my_row) : 0.f;

    // ---- the entries, thread tid's at tid + 512 e of the slice, and their largest magnitude
    Bits top = 0;
    auto put = [&](uint32_t k, Entry v) {
        if (k < padded) entries[k] = v;
        const Bits m = (Bits)FloatBits<Entry>::magnitude(v);
        top = m > top ? m : top;
    };
    if (!kFinal && p.norm_w) {
        // a normed plan (at most 4096 entries, one CTA over them): the norm as rmsnorm_kernel forms it (512 threads,
        // element i of a thread's eight is tid + 512 i, warp sums by shuffles, then the warps' sums in order)
        const float *xs = static_cast<const float *>(p.in), *rs = p.in_residual ? p.in_residual : xs;
        const bool writer = p.x_out && blockIdx.x == 0;
        float hx[8], hr[8], nw[8], sc[8], ss = 0.f;
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const uint32_t i = min(tid + e * kSumThreads, n_bits - 1);
            nw[e] = __ldg(p.norm_w + i);
            sc[e] = p.in_scale ? __ldg(p.in_scale + i) : 1.f;
        }
        qk::pdl_wait();
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const uint32_t i = min(tid + e * kSumThreads, n_bits - 1);
            hx[e] = __ldcg(xs + i);
            hr[e] = __ldcg(rs + i);
        }
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const uint32_t i = tid + e * kSumThreads;
            float h = hx[e];
            if (p.in_residual) h += hr[e];
            if (writer && i < n_bits) p.x_out[i] = h;
            if (kRoundBf16) h = round_bf16_fast(h);
            hx[e] = i < n_bits ? h : 0.f;
            ss += hx[e] * hx[e];
        }
        for (int off = 16; off > 0; off >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, off);
        if (lane == 0) norm_red[warp] = ss;
        __syncthreads();
        float total = 0.f;
#pragma unroll
        for (int w = 0; w < kWarps; w += 4) {
            const float4 r = *reinterpret_cast<const float4 *>(norm_red + w);
            total += r.x;
            total += r.y;
            total += r.z;
            total += r.w;
        }
        const float inv = 1.0f / sqrtf(total / (float)n_bits + p.norm_eps);
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            float x = hx[e] * inv * nw[e];
            if (kRoundBf16) x = round_bf16_fast(x);
            if (p.in_scale) x = sc[e] * x;
            if (kRoundBf16) x = round_bf16_fast(x);
            put(tid + e * kSumThreads, (Entry)(tid + e * kSumThreads < n_bits ? x : 0.f));
        }
    } else {
        using T = typename std::conditional<kFinal, double, float>::type;
        constexpr int kLoad = kFinal ? 4 : 8;
        qk::pdl_wait();
#pragma unroll 1
        for (uint32_t k0 = tid; k0 < padded; k0 += kLoad * kSumThreads) {
            T vals[kLoad];
            load_inputs<kFinal, kRoundBf16, kLoad, T>(p, [&](int e) { return k_lo + k0 + e * kSumThreads; }, max(1u, k_hi),
                                                      k_hi > k_lo, vals);
#pragma unroll
            for (int e = 0; e < kLoad; ++e) put(k0 + e * kSumThreads, (Entry)vals[e]);
        }
    }
    if constexpr (sizeof(Entry) == 4) {
        top = __reduce_max_sync(0xffffffffu, top);
    } else {
        for (int off = 16; off > 0; off >>= 1) {
            const Bits other = __shfl_xor_sync(0xffffffffu, top, off);
            top = other > top ? other : top;
        }
    }
    if (lane == 0) top_red[warp] = top;
    __syncthreads();
    top = top_red[lane % kWarps];
    if constexpr (sizeof(Entry) == 4) {
        top = __reduce_max_sync(0xffffffffu, top);
    } else {
        for (int off = kWarps / 2; off > 0; off >>= 1) {
            const Bits other = __shfl_xor_sync(0xffffffffu, top, off);
            top = other > top ? other : top;
        }
    }

    if (n_rank > 1) {  // the whole vector's largest: every CTA tells every other, once that one has begun
        asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
        if (tid < n_rank) {
            uint32_t there;
            asm volatile("mapa.shared::cluster.u32 %0, %1, %2;"
                         : "=r"(there)
                         : "r"((uint32_t)__cvta_generic_to_shared(peer_top + rank)), "r"(tid));
            if constexpr (sizeof(Entry) == 4) asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(there), "r"(top) : "memory");
            else asm volatile("st.shared::cluster.u64 [%0], %1;" ::"r"(there), "l"(top) : "memory");
        }
        __syncwarp();
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
        for (uint32_t c = 0; c < n_rank; ++c) top = peer_top[c] > top ? peer_top[c] : top;
    }

    // ---- the entries on the grid of the largest one.  x = v * 2^(shift - 21) lies within 2^26; q = rint(x * 2^21) =
    // hi * 2^21 + lo with hi = rint(x), exactly.
    const bool nonfinite = top >= FloatBits<Entry>::kBad;  // a NaN or an infinity: every row is NaN, as in the digit forms
    const FixedPoint fp = fixed_point_of(nonfinite ? 0.0 : FloatBits<Entry>::as_double(top));
    const int down = fp.shift - kSumLow;
    if (sizeof(Entry) == 4 && down <= 127) {  // (always down > -126: a float32 is below 2^128)
        const float scale = nonfinite ? 0.f : __uint_as_float((uint32_t)(127 + down) << 23);
#pragma unroll 2
        for (uint32_t k = tid; k < padded; k += kSumThreads) {
            const float x = nonfinite ? 0.f : (float)entries[k] * scale, n = rintf(x);
            const uint32_t at = k % kSumEntries * z_pitch + k / kSumEntries;
            zh[at] = (int)n;
            zl[at] = __float2int_rn((x - n) * (float)(1 << kSumLow));
        }
    } else {
#pragma unroll 1
        for (uint32_t k = tid; k < padded; k += kSumThreads) {
            const long long q = nonfinite ? 0 : fp.quant((double)entries[k]);
            const int hi = (int)((q + (1ll << (kSumLow - 1))) >> kSumLow);
            const uint32_t at = k % kSumEntries * z_pitch + k / kSumEntries;
            zh[at] = hi;
            zl[at] = (int)(q - ((long long)hi << kSumLow));
        }
    }
    cp_async_wait<0>();
    __syncthreads();

    // ---- the sums over the set bits.  A thread's sum of hi stays within 2^30, of lo within 2^24: over the lanes hi goes in
    // two halves.
    auto over_warp = [&](int h, int r, bool rests) {
        const int top_half = __reduce_add_sync(0xffffffffu, h >> 15), low_half = __reduce_add_sync(0xffffffffu, h & 0x7fff);
        long long q = (((long long)top_half << 15) + low_half) << kSumLow;
        if (rests) q += __reduce_add_sync(0xffffffffu, r);
        return q;
    };
    const uint32_t groups = kWarps / lay.warps, group = warp / lay.warps, vw = warp % lay.warps;
    if (group < groups) {
        const uint32_t l = vw * 32 + lane;
        int hi[kSumEntries], lo[kSumEntries], h_all = 0, r_all = 0;
        bool rest = false;
#pragma unroll
        for (int j = 0; j < kSumEntries; ++j) {
            hi[j] = zh[j * z_pitch + l];
            lo[j] = zl[j * z_pitch + l];
            rest |= lo[j] != 0;
            h_all += hi[j];
            r_all += lo[j];
        }
        const bool rests = __any_sync(0xffffffffu, rest) != 0;
        if (group == 0) {
            const long long total = over_warp(h_all, r_all, rests);
            if (lane == 0) part[rows_per_block * lay.warps + vw] = total;
        }
        const uint8_t *w = slab + l * (kSumEntries / 8);
        if (rests) {
#pragma unroll 2
            for (uint32_t row = group; row < rows; row += groups) {
                const uint32_t bits = *reinterpret_cast<const uint16_t *>(w + row * lay.pitch);
                int h = 0, r = 0;
#pragma unroll
                for (int j = 0; j < kSumEntries; ++j)
                    asm("{\n .reg .pred p;\n .reg .b32 t;\n and.b32 t, %4, %5;\n setp.ne.u32 p, t, 0;\n"
                        " @p add.s32 %0, %0, %2;\n @p add.s32 %1, %1, %3;\n}"
                        : "+r"(h), "+r"(r)
                        : "r"(hi[j]), "r"(lo[j]), "r"(bits), "r"(1u << j));
                const long long q = over_warp(h, r, true);
                if (lane == 0) part[row * lay.warps + vw] = q;
            }
        } else {
#pragma unroll 4
            for (uint32_t row = group; row < rows; row += groups) {
                const uint32_t bits = *reinterpret_cast<const uint16_t *>(w + row * lay.pitch);
                int h = 0;
#pragma unroll
                for (int j = 0; j < kSumEntries; ++j)
                    asm("{\n .reg .pred p;\n .reg .b32 t;\n and.b32 t, %2, %3;\n setp.ne.u32 p, t, 0;\n"
                        " @p add.s32 %0, %0, %1;\n}"
                        : "+r"(h)
                        : "r"(hi[j]), "r"(bits), "r"(1u << j));
                const long long q = over_warp(h, 0, false);
                if (lane == 0) part[row * lay.warps + vw] = q;
            }
        }
    }
    __syncthreads();

    // ---- rows: the warps' parts, the sign sum, the stage's epilogue
    const int oexp = -fp.shift;
    const double unit = oexp > -1000 && oexp < 1000 ? __hiloint2double((1023 + oexp) << 20, 0) : 0.0;
    long long total = 0;
    for (uint32_t w = 0; w < lay.warps; ++w) total += part[rows_per_block * lay.warps + w];
    auto row_value = [&](uint32_t r) {
        long long s = 0;
        for (uint32_t w = 0; w < lay.warps; ++w) s += part[r * lay.warps + w];
        return 2 * s - total;
    };
    auto finish = [&](uint32_t r, long long sum) {
        const uint32_t row = row0 + r;
        const double n = (double)sum;
        double val = nonfinite ? nan("") : unit != 0.0 ? n * unit : ldexp(n, oexp);
        if (kRoundBf16) val = (double)round_bf16((float)val);
        if (kFinal) {
            // (each thread's first row has its scale and bias at hand)
            const bool first = n_rank == 1 && r < kSumThreads;
            float y = (float)val;
            if (p.out_scale) y = __fmul_rn(y, first ? row_scale : p.out_scale[row]);  // (rounded before the bias is
            if (p.out_bias) y = __fadd_rn(y, first ? row_bias : p.out_bias[row]);     // added, as everywhere)
            static_cast<float *>(p.out)[row] = y;
        } else {
            static_cast<double *>(p.out)[row] = val;
        }
    };
    if (n_rank == 1) {
#pragma unroll 1
        for (uint32_t r = tid; r < rows; r += kSumThreads) finish(r, row_value(r));
        return;
    }
#pragma unroll 1
    for (uint32_t r = tid; r < rows; r += kSumThreads) row_sum[r] = row_value(r);
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
#pragma unroll 1
    for (uint32_t r = rank + n_rank * tid; r < rows; r += n_rank * kSumThreads) {
        long long sum = 0;
        for (uint32_t c = 0; c < n_rank; ++c) {
            // (row_sum lies where the slice's width puts it: the last CTA's may be narrower than the others')
            const uint32_t lo = min(c * slice_bits, n_bits), hi = min(lo + slice_bits, n_bits);
            const uint32_t at = (uint32_t)__cvta_generic_to_shared(smem_dyn) +
                                sum_layout(max(1u, hi - lo), rows_per_block, sizeof(Entry)).row_sum + 8 * r;
            uint32_t there;
            long long one;
            asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(there) : "r"(at), "r"(c));
            asm volatile("ld.shared::cluster.s64 %0, [%1];" : "=l"(one) : "r"(there) : "memory");
            sum += one;
        }
        finish(r, sum);
    }
    // (nobody leaves while a peer may still read its sums)
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

__device__ __forceinline__ void sum_cluster(uint32_t &rank, uint32_t &n_rank) {
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(n_rank));
}
template <bool kRoundBf16, bool kFinal>
__global__ void __launch_bounds__(kSumThreads, 1)
gemv_sum_kernel(const StageParams *__restrict__ many, uint32_t rows_per_block, uint32_t slice_bits) {
    qk::pdl_launch();
    uint32_t rank, n_rank;
    sum_cluster(rank, n_rank);
    const StageParams p = many[blockIdx.y];
    sum_form<kRoundBf16, kFinal>(p, rows_per_block, slice_bits, rank, n_rank);
}
template <bool kRoundBf16, bool kFinal>
__global__ void __launch_bounds__(kSumThreads, 1)
gemv_sum_run_kernel(const __grid_constant__ StageRun run, uint32_t rows_per_block, uint32_t slice_bits) {
    qk::pdl_launch();
    uint32_t rank, n_rank;
    sum_cluster(rank, n_rank);
    const StageParams p = run_params(run, blockIdx.y);
    sum_form<kRoundBf16, kFinal>(p, rows_per_block, slice_bits, rank, n_rank);
}

}  // namespace
