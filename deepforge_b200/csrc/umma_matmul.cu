// Matrix products on the 5th-generation tensor cores for every extent: C = steps(A B), A [M, K] with K contiguous, B with
// K or N contiguous, 16-bit floats (bf16, f16), FP8 codes (MATMUL_FP8) or FP8 codes with E8M0 block scales (MXFP8).
//
// kPieces: f32 operands as three bf16 pieces each (split_f32.cu), six products of a K block's tiles per stage: every piece is copied
// once for two products (six-fold deep copies moved and stored twice as much: 1183 x 1888 x 5360 154 us then, 128 now, 87 of
// products; 4096^3 586 of 500).
//
// kSummed: 16-bit operands, f32 C, the products of every K block in an accumulator of their own and the blocks added by the epilogue in
// f32. The tensor cores cut off what a sum does not hold, toward zero, so that the error of one long accumulation grows with K:
// 2050 x 8184 x 1040 bf16 to f32 is 9.1e-6 from 64 bits in one accumulator, 9.6e-7 by the CUDA cores' additions, 2.2e-7 this way. The
// forms that ran there (or in the one-launch f32 kernel) keep an accuracy no worse than theirs. The epilogue's two loads and 64
// additions a block set the pace: 4096 x 4104 x 4104 124 us in one accumulator, 234 this way, 9227 on the CUDA cores.
// kCodesSummed: the same for FP8 codes. kScaledSummed: for block-scaled codes (1026 x 8160 x 1040 to f32: 1.2e-7 on the CUDA cores, 4.7e-7 in one accumulator).
//
// Extents are free because the copies are: TMA fills what lies outside a matrix with zeros and clips what would be stored
// there, so a tile may hang over any edge. Only the rows' starts have to fall on 16-byte boundaries.
//
// Three shapes of work, one kernel body:
//   CG = 2      two SMs (a cluster) on one 256 x bn tile: CTA r holds rows 128 r .. 128 r + 127 of A and half of the bn columns
//               of B, and one thread of CTA 0 issues tcgen05.mma.cta_group::2, which reads both. Each operand byte is written
//               to shared memory once and read once, and both go through the same 128 B per clock: a 128 x 256 x 64 step of
//               ONE SM moves 2 x 48 KB = 768 clocks for 512 clocks of products, the pair moves 2 x 32 KB = 512 per SM.
//   CG = 1      one SM per 128 x bn tile, for problems whose tiles are few.
//   splits > 1  CG = 1, and a cluster of `splits` CTAs shares out the K blocks of ONE tile; the partial tiles meet through
//               distributed shared memory and are added in rank order. For products with fewer tiles than SMs.
// bn is 64, 128, 192 or 256 at run time; choose_shape() says which shape a product takes and why.
//
// Warps: 0 loads (TMA), 1 issues products, 4-11 are the epilogue (two groups of four, alternating 128-byte column boxes), and
// with block scales 2, 3 and 12-15 gather them. Two accumulators in tensor memory, so that a tile's epilogue
// runs under the next tile's products. Finished boxes leave through a swizzled staging tile by TMA; a thread's own row of
// 64 bytes at a row's distance would jam the load/store unit.
#include <algorithm>

#include "matmul_shape.cuh"
#include "umma.cuh"
#include "umma_ptx.cuh"

namespace dfgpu {
namespace {

template <int KIND> constexpr bool kHasScales = KIND == kScaled || KIND == kScaledSummed;
template <int KIND> constexpr bool kInRegisters = KIND == kSummed || KIND == kCodesSummed;
template <int KIND> constexpr bool kInPlace = KIND == kScaledSummed || KIND == kPiecesSummed;   // ... in tensor memory
template <int KIND> constexpr bool kInBlocks = kInRegisters<KIND> || kInPlace<KIND>;
template <int KIND> constexpr bool kHasPieces = KIND == kPieces || KIND == kPiecesSummed;   // an accumulator per K block, summed by the epilogue
enum { kStepRelu = 1, kStepBias = 2, kStepFull = 3 };

struct TileArgs {
    int32_t m_total, n_total;
    int32_t m_tiles, k_blocks;
    int32_t bn;                       // columns of a tile
    int32_t whole_items, items;       // work items: whole tiles, and after them the halves of the tiles that are left for the last round
    int32_t splits, k_per_split;
    int32_t stages, stage_bytes;
    int32_t blocks_per_sum, sums_column;             // kInBlocks: K blocks of an accumulator; kInPlace: tensor-memory column of the sums
    int32_t acc_stride, acc_shift, scale_columns;   // tensor memory: see launch_problem(); 1 << acc_shift accumulators
    int32_t a_bytes;                  // A of one CTA and stage; B lies behind it
    int32_t b_box_bytes, b_box_columns;   // B comes in boxes
    int32_t b_mn_major;
    int32_t a_piece_rows, b_piece_rows;   // kPieces: rows of the maps from one piece to the next
    uint32_t idesc;
    int32_t staging_offset, barrier_offset;
    int32_t staging_boxes;            // per epilogue group, used in turn: 1 or 2
    void* out;
    int64_t out_ld;
    int32_t out_dtype;
    int32_t tma_store;                // C's rows start on 16-byte boundaries
    int32_t step_count;
    int32_t step_kind[kMaxSteps], step_dtype[kMaxSteps], step_vector[kMaxSteps];
    float relu_lower[kMaxSteps], relu_upper[kMaxSteps], relu_slope[kMaxSteps];
    const void* step_data[kMaxSteps];
    int64_t step_ld[kMaxSteps];
    // MATMUL_FP8: value = acc * *descale_a * *descale_b, *amax_bits = max |value| (bits of the non-negative f32, NaN
    // canonical), C = value * *scale_c
    const float* descale_a;
    const float* descale_b;
    const float* scale_c;
    unsigned int* amax_bits;
    // block scales: [M, K/32] and [K/32, N], one byte each
    const uint8_t* sfa;
    const uint8_t* sfb;
    int64_t sfa_ld, sfb_ld;
    int32_t scale_blocks, sfa_words;  // K / 32; sfa rows are whole aligned words
};

// ---- cluster and pair forms of the PTX wrappers ------------------------------------------------------------

__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
// ... which waits for no store of the thread's own: for threads that have only read the others' memory, and have what they read
__device__ __forceinline__ void cluster_arrive_relaxed() { asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ uint32_t address_in(uint32_t own_address, uint32_t rank) {
    uint32_t remote;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(own_address), "r"(rank));
    return remote;
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_address) {
    // (tensor memory is handed over, which the tcgen05 fences order, or block scales behind a proxy fence: see the scale loaders; released to
    // the cluster, it would wait for all stores)
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_address) : "memory");
}
__device__ __forceinline__ float4 load_from_rank(uint32_t cluster_address) {
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(cluster_address) : "memory");
    return v;
}
template <int CG>
__device__ __forceinline__ void load_tile(uint32_t dst, const CUtensorMap* map, int c0, int c1, uint32_t bar) {
    if constexpr (CG == 2)
        asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                     ::"r"(dst), "l"(map), "r"(c0), "r"(c1), "r"(bar) : "memory");
    else tma_load_2d(dst, map, c0, c1, bar);
}
// Arrival on a barrier of this CTA, and with CG = 2 on the same barrier of the other one.
template <int CG>
__device__ __forceinline__ void commit_to_all(uint32_t bar) {
    if constexpr (CG == 2) {
        const uint16_t both = 3;
        asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar), "h"(both) : "memory");
    } else {
        umma_commit(bar);
    }
}
template <int CG>
__device__ __forceinline__ void alloc_columns(uint32_t slot) {
    if constexpr (CG == 2) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    } else {
        tmem_alloc(slot, 512);
        tmem_relinquish();
    }
}
template <int CG>
__device__ __forceinline__ void free_columns(uint32_t base) {
    if constexpr (CG == 2) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(base), "r"(512u) : "memory");
    else tmem_dealloc(base, 512);
}
template <int KIND, int CG>
__device__ __forceinline__ void product(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate, uint32_t sfa, uint32_t sfb) {
#define DFGPU_MMA(FORM)                                                                                                   \
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma." FORM " [%0], %1, %2, %3, p;\n\t}"          \
                 ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate) : "memory")
    constexpr bool sixteen = KIND == kSixteen || kHasPieces<KIND> || KIND == kSummed;
    if constexpr (sixteen && CG == 1) DFGPU_MMA("cta_group::1.kind::f16");
    if constexpr (sixteen && CG == 2) DFGPU_MMA("cta_group::2.kind::f16");
    if constexpr ((KIND == kCodes || KIND == kCodesSummed) && CG == 1) DFGPU_MMA("cta_group::1.kind::f8f6f4");
    if constexpr ((KIND == kCodes || KIND == kCodesSummed) && CG == 2) DFGPU_MMA("cta_group::2.kind::f8f6f4");
#undef DFGPU_MMA
#define DFGPU_MMA(FORM)                                                                                                   \
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma." FORM ".kind::mxf8f6f4.block_scale [%0], %1, %2, %3, [%5], [%6], p;\n\t}" \
                 ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate), "r"(sfa), "r"(sfb) : "memory")
    if constexpr (kHasScales<KIND> && CG == 1) DFGPU_MMA("cta_group::1");
    if constexpr (kHasScales<KIND> && CG == 2) DFGPU_MMA("cta_group::2");
#undef DFGPU_MMA
}
// 32 rows x 16 bytes of shared memory -> 4 columns of tensor memory, replicated to the four lane quarters.
// (CG = 2: each CTA's from its own shared memory.)
template <int CG>
__device__ __forceinline__ void copy_scales(uint32_t tmem_dst, uint32_t address) {
    // an unswizzled K-major block: 8-row groups 128 bytes apart
    const uint64_t desc = static_cast<uint64_t>((address & 0x3FFFFu) >> 4) | (static_cast<uint64_t>(128u >> 4) << 32) | (1ull << 46);
    if constexpr (CG == 2) asm volatile("tcgen05.cp.cta_group::2.32x128b.warpx4 [%0], %1;" ::"r"(tmem_dst), "l"(desc) : "memory");
    else asm volatile("tcgen05.cp.cta_group::1.32x128b.warpx4 [%0], %1;" ::"r"(tmem_dst), "l"(desc) : "memory");
}

// ---- the fused steps on values of one row of C ---------------------------------------------------------------

__device__ __forceinline__ void widen_pair(uint32_t word, int dtype, float& lo, float& hi) {
    if (dtype == DFGPU_BF16) {
        lo = __uint_as_float(word << 16);
        hi = __uint_as_float(word & 0xffff0000u);
    } else {
        const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&word));
        lo = f.x;
        hi = f.y;
    }
}
// The fused ADD operands: COUNT neighbouring columns from element `first` on, as far as the row reaches (`live` of them). Every load
// is issued before the first use, whole rows in 16-byte units where COUNT allows: a load at a time, each behind a branch on the
// type, took an epilogue part of 32 columns 8 (ragged edges: 32) trips to the L2 one after the other, 3 to 8 us of a launch with a
// bias (238 x 312 x 304 bf16 with bias and ReLU: 10.2 us that way, 6.0 now, 4.9 without either).
template <int COUNT>
__device__ __forceinline__ void load_words(uint32_t (&words)[COUNT / 2], const uint16_t* p, int live, bool vector) {   // 16-bit operands
    if (vector && live >= COUNT) {
        if constexpr (COUNT % 8 == 0) {
#pragma unroll
            for (int j = 0; j < COUNT / 8; ++j) {
                const uint4 q = reinterpret_cast<const uint4*>(p)[j];
                words[4 * j] = q.x;
                words[4 * j + 1] = q.y;
                words[4 * j + 2] = q.z;
                words[4 * j + 3] = q.w;
            }
        } else {
#pragma unroll
            for (int j = 0; j < COUNT / 4; ++j) {
                const uint2 q = reinterpret_cast<const uint2*>(p)[j];
                words[2 * j] = q.x;
                words[2 * j + 1] = q.y;
            }
        }
    } else {
        uint16_t halves[COUNT];
#pragma unroll
        for (int i = 0; i < COUNT; ++i) halves[i] = i < live ? p[i] : 0;
#pragma unroll
        for (int i = 0; i < COUNT / 2; ++i) words[i] = halves[2 * i] | (static_cast<uint32_t>(halves[2 * i + 1]) << 16);
    }
}
template <int COUNT>
__device__ __forceinline__ void add_words(float (&v)[COUNT], const uint32_t (&words)[COUNT / 2], int dtype) {
#pragma unroll
    for (int i = 0; i < COUNT / 2; ++i) {
        float lo, hi;
        widen_pair(words[i], dtype, lo, hi);
        v[2 * i] = __fadd_rn(v[2 * i], lo);
        v[2 * i + 1] = __fadd_rn(v[2 * i + 1], hi);
    }
}
// (32-bit operands BATCH loads at a time: where a row's sums are in registers too, 32 more spill)
template <int COUNT, int BATCH>
__device__ __forceinline__ void add_operand(float (&v)[COUNT], const void* data, int dtype, int64_t first, int live, bool vector) {
    if (dtype != DFGPU_F32) {
        uint32_t words[COUNT / 2];
        load_words<COUNT>(words, static_cast<const uint16_t*>(data) + first, live, vector);
        add_words<COUNT>(v, words, dtype);
        return;
    }
    const float* p = static_cast<const float*>(data) + first;
#pragma unroll
    for (int at = 0; at < COUNT; at += BATCH) {
        float x[BATCH];
        if (vector && live >= COUNT) {
#pragma unroll
            for (int j = 0; j < BATCH / 4; ++j) {
                const float4 q = reinterpret_cast<const float4*>(p + at)[j];
                x[4 * j] = q.x;
                x[4 * j + 1] = q.y;
                x[4 * j + 2] = q.z;
                x[4 * j + 3] = q.w;
            }
        } else {
#pragma unroll
            for (int i = 0; i < BATCH; ++i) x[i] = at + i < live ? p[at + i] : 0.0f;
        }
#pragma unroll
        for (int i = 0; i < BATCH; ++i) v[at + i] = __fadd_rn(v[at + i], x[i]);
    }
}

struct Scalars {
    float descale_a, descale_b, scale_c;
    float magnitude;   // largest |value| of this thread so far (NaN sticks)
    // finite de-scales: `magnitude` is that of the accumulators, which they are applied to once, at the end. (Products with them and their roundings
    // keep the order of magnitudes, and an infinity times zero is a NaN then as it would have been.)
    bool at_end;
};
template <bool CODES>
__device__ __forceinline__ Scalars load_scalars(const TileArgs& args) {
    Scalars s{};
    if constexpr (CODES) {
        s.descale_a = *args.descale_a;
        s.descale_b = *args.descale_b;
        s.scale_c = *args.scale_c;
        s.at_end = fabsf(s.descale_a) < INFINITY && fabsf(s.descale_b) < INFINITY;
    }
    return s;
}
template <bool CODES>
__device__ __forceinline__ void fold_amax(const TileArgs& args, const Scalars& s, int lane, bool ok) {
    if constexpr (!CODES) return;
    const float magnitude = s.at_end ? fabsf(__fmul_rn(__fmul_rn(s.magnitude, s.descale_a), s.descale_b)) : s.magnitude;
    unsigned int bits = magnitude != magnitude ? 0x7fc00000u : __float_as_uint(magnitude);
    bits = __reduce_max_sync(0xffffffffu, bits);
    if (lane == 0 && bits != 0u && ok) atomicMax(args.amax_bits, bits);
}

// COUNT neighbouring columns of one row: fused steps, then MATMUL_FP8's scalars. `row_live`: the row exists. `ahead`: the first
// step's operand, where it was loaded ahead.
// CODES: MATMUL_FP8, which has the scalars and no steps; the others have none of the scalars (neither is compiled into the other's kernel).
template <bool CODES, int BATCH, int COUNT>
__device__ __forceinline__ void apply_steps(const TileArgs& args, float (&v)[COUNT], int row, int col0, bool row_live, Scalars& scalars, const uint32_t (*ahead)[COUNT / 2] = nullptr) {
    const int live = args.n_total - col0;
    if constexpr (!CODES) {
        if (ahead != nullptr) add_words<COUNT>(v, *ahead, args.step_dtype[0]);
        for (int s = ahead != nullptr ? 1 : 0; s < args.step_count; ++s) {
            const int kind = args.step_kind[s];
            if (kind == kStepRelu) {
                relu_values(v, args.relu_lower[s], args.relu_upper[s], args.relu_slope[s], row_live);
            } else if (kind == kStepBias || row_live) {
                add_operand<COUNT, BATCH>(v, args.step_data[s], args.step_dtype[s], (kind == kStepBias ? 0 : row * args.step_ld[s]) + col0, live, args.step_vector[s] != 0);
            }
        }
    }
    if constexpr (CODES) {
        // value = (sum + 0) * descale_a * descale_b, C = value * scale_c, each rounded by itself, two at a time. (+0.0 first: the reference's
        // sum starts from +0.0 and so is never -0.0, the tensor core's can be.) Where an epilogue is not hidden its instructions are what a
        // tile waits for.
        const uint64_t by_a = pack2(scalars.descale_a, scalars.descale_a), by_b = pack2(scalars.descale_b, scalars.descale_b), by_c = pack2(scalars.scale_c, scalars.scale_c);
        float top = 0.0f;
#pragma unroll
        for (int e = 0; e < COUNT; e += 2) {
            const uint64_t value = mul2(mul2(add2(pack2(v[e], v[e + 1]), 0ull), by_a), by_b);
            float lo = v[e], hi = v[e + 1];
            if (!scalars.at_end) unpack2(value, lo, hi);
            if (live < COUNT) {
                lo = e < live ? lo : 0.0f;
                hi = e + 1 < live ? hi : 0.0f;
            }
            asm("max.NaN.abs.f32 %0, %0, %1, %2;" : "+f"(top) : "f"(lo), "f"(hi));
            unpack2(mul2(value, by_c), v[e], v[e + 1]);
        }
        if (row_live) scalars.magnitude = maximum_nan(scalars.magnitude, top);
    }
}

// The first step's operand for 32 columns, where it is 16 bits wide.
__device__ __forceinline__ void load_ahead(const TileArgs& args, uint32_t (&words)[16], int row, int col0, bool row_live) {
    const bool per_column = args.step_kind[0] == kStepBias;
    load_words<32>(words, static_cast<const uint16_t*>(args.step_data[0]) + (per_column ? 0 : row * args.step_ld[0]) + col0, per_column || row_live ? args.n_total - col0 : 0,
                   args.step_vector[0] != 0);
}

__device__ __forceinline__ uint32_t narrow_pair(float lo, float hi, int dtype) {
    if (dtype == DFGPU_BF16) {
        const __nv_bfloat162 pair = __floats2bfloat162_rn(lo, hi);
        return *reinterpret_cast<const uint32_t*>(&pair);
    }
    const __half2 pair = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&pair);
}
__device__ __forceinline__ uint32_t encode_four_e4m3(const float* f) {
    uint32_t lo = encode_e4m3_pair(f[0], f[1]), hi = encode_e4m3_pair(f[2], f[3]);
    // NaN -> 0x7f whatever its sign (the hardware convert keeps the sign bit)
    if (f[0] != f[0]) lo = (lo & 0xff00u) | 0x7fu;
    if (f[1] != f[1]) lo = (lo & 0x00ffu) | 0x7f00u;
    if (f[2] != f[2]) hi = (hi & 0xff00u) | 0x7fu;
    if (f[3] != f[3]) hi = (hi & 0x00ffu) | 0x7f00u;
    return lo | (hi << 16);
}

// Four neighbouring columns straight to C (the split form: neighbouring threads hold neighbouring columns).
__device__ __forceinline__ void store_four(const TileArgs& args, const float (&v)[4], int row, int col) {
    const int64_t at = row * args.out_ld + col;
    const int live = args.n_total - col;
    if (live >= 4 && args.tma_store) {
        if (args.out_dtype == DFGPU_F32) *reinterpret_cast<float4*>(static_cast<float*>(args.out) + at) = make_float4(v[0], v[1], v[2], v[3]);
        else if (args.out_dtype == DFGPU_E4M3) *reinterpret_cast<uint32_t*>(static_cast<uint8_t*>(args.out) + at) = encode_four_e4m3(v);
        else *reinterpret_cast<uint2*>(static_cast<uint16_t*>(args.out) + at) = make_uint2(narrow_pair(v[0], v[1], args.out_dtype), narrow_pair(v[2], v[3], args.out_dtype));
        return;
    }
    for (int i = 0; i < 4; ++i)
        if (i < live) store_from_f32(args.out, args.out_dtype, at + i, v[i]);
}

template <bool CLUSTER>
__device__ __forceinline__ bool wait_warp(uint32_t bar, uint32_t parity, int code) {
    if constexpr (CLUSTER) return mbar_wait_warp_cluster(bar, parity, code);
    else return mbar_wait_warp<true>(bar, parity, code);
}

// kPieces: 32 columns of the products of the lower pieces onto those of the leading ones.
__device__ __forceinline__ void add_small_products(uint32_t address, uint32_t (&sum)[32]) {
    uint32_t small[32];
    tmem_load_32(address, small);
    tmem_load_wait();
#pragma unroll
    for (int e = 0; e < 32; ++e) sum[e] = __float_as_uint(__fadd_rn(__uint_as_float(sum[e]), __uint_as_float(small[e])));
}

__device__ __forceinline__ void tmem_put_32(uint32_t address, const uint32_t (&r)[32]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
                 ::"r"(address), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31]) : "memory");
}
// kSummed, kCodesSummed: this thread's row of a tile, the boxes g and g + 2 of 32 columns, summed over the K blocks of the walk. `local` counts
// accumulators, as the issuing warp does; one is handed back as soon as it is in registers.
template <int CG>
__device__ __forceinline__ void sum_blocks(float (&sums)[2][32], uint32_t columns, int acc_stride, int boxes, int g, int blocks, int& local, uint32_t acc_full, uint32_t acc_empty,
                                           int lane, bool& ok) {
    for (int block = 0; block < blocks; ++block, ++local) {
        const int acc = local & 1;
        if (ok) ok = mbar_wait_warp<true>(acc_full + 8u * acc, (local >> 1) & 1, 585);   // (the warp stays together)
        tc_fence_after();
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            if (q == 1 && g + 2 >= boxes) break;   // (two boxes at least: one for each group)
            uint32_t raw[32];
            tmem_load_32(columns + acc * acc_stride + (g + 2 * q) * 32, raw);
            tmem_load_wait();
#pragma unroll
            for (int e = 0; e < 32; ++e) asm volatile("" : "+r"(raw[e]));   // (no use above the wait)
#pragma unroll
            for (int e = 0; e < 32; ++e) sums[q][e] = block == 0 ? __uint_as_float(raw[e]) : __fadd_rn(sums[q][e], __uint_as_float(raw[e]));
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) {
            if (CG == 2) mbar_arrive_cluster(acc_empty + 8u * acc);
            else mbar_arrive(acc_empty + 8u * acc);
        }
    }
}

// The same with the sums in tensor memory, behind the accumulators: kScaledSummed's 16 warps leave too few registers, and kPiecesSummed
// adds the products of the lower pieces on the way.
template <int KIND, int CG>
__device__ __forceinline__ void sum_blocks_in_place(const TileArgs& args, uint32_t columns, int boxes, int g, int blocks, int& local, uint32_t acc_full, uint32_t acc_empty, int lane, bool& ok) {
    for (int block = 0; block < blocks; block += args.blocks_per_sum, ++local) {
        const int acc = local & args.acc_shift;
        if (ok) ok = mbar_wait_warp<true>(acc_full + 8u * acc, (local >> args.acc_shift) & 1, KIND == kPiecesSummed ? 565 : 595);
        tc_fence_after();
        for (int box = g; box < boxes; box += 2) {
            const uint32_t own = columns + acc * args.acc_stride + box * 32, target = columns + args.sums_column + box * 32;
            uint32_t raw[32];
            tmem_load_32(own, raw);
            tmem_load_wait();
#pragma unroll
            for (int e = 0; e < 32; ++e) asm volatile("" : "+r"(raw[e]));   // (no use above the wait)
            if constexpr (KIND == kPiecesSummed) add_small_products(own + args.bn, raw);
            if (block > 0) add_small_products(target, raw);   // (the sum so far)
            tmem_put_32(target, raw);
        }
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        tc_fence_before();
        __syncwarp();
        if (lane == 0) {
            if (CG == 2) mbar_arrive_cluster(acc_empty + 8u * acc);
            else mbar_arrive(acc_empty + 8u * acc);
        }
    }
}

template <int KIND>
constexpr int thread_count() { return kHasScales<KIND> ? 512 : 384; }

// One K block's scales of a tile as a lane reads them from the plain tensors: 4 rows of A (rows lane, lane + 32, ... of 128)
// and 4 or 8 columns of B, four K blocks each. Addresses are clamped, so that nothing branches around a load and all of
// them are in flight together (with branches the gather took three times as long as the products); pack() selects. The
// loads of a warp's next block are issued before it waits for its current slot, and packed after.
struct RawScales {
    uint32_t a[4];          // words, or bytes of block 0 when rows cannot be read as words
    uint32_t a_more[4][3];  // bytes of blocks 1..3 then
    uint32_t b[2][4][4];
};
__device__ __forceinline__ void load_scales(const TileArgs& args, int row0, int col0, int kb, int lane, RawScales& raw) {
    const int first = kb * 4, last = args.scale_blocks - 1;
    if (args.sfa_words) {
#pragma unroll
        for (int g = 0; g < 4; ++g)
            raw.a[g] = *reinterpret_cast<const uint32_t*>(args.sfa + min(row0 + g * 32 + lane, args.m_total - 1) * args.sfa_ld + first);
    } else {
#pragma unroll
        for (int g = 0; g < 4; ++g) {
            const uint8_t* p = args.sfa + min(row0 + g * 32 + lane, args.m_total - 1) * args.sfa_ld;
            raw.a[g] = p[first];
#pragma unroll
            for (int j = 1; j < 4; ++j) raw.a_more[g][j - 1] = p[min(first + j, last)];
        }
    }
    const uint8_t* base[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) base[j] = args.sfb + min(first + j, last) * args.sfb_ld;
#pragma unroll
    for (int c = 0; c < 2; ++c) {
        if (c == 1 && args.bn <= 128) break;
#pragma unroll
        for (int g = 0; g < 4; ++g) {
            const int col = min(col0 + c * 128 + g * 32 + lane, args.n_total - 1);
#pragma unroll
            for (int j = 0; j < 4; ++j) raw.b[c][g][j] = base[j][col];
        }
    }
}
// The words tcgen05.cp wants: byte j the scale of K block j. Blocks, rows and columns past the end count as 2^0 (their codes
// are zeros).
__device__ __forceinline__ uint32_t pack_word(uint32_t b0, uint32_t b1, uint32_t b2, uint32_t b3, int live) {
    return b0 | ((live > 1 ? b1 : 0x7fu) << 8) | ((live > 2 ? b2 : 0x7fu) << 16) | ((live > 3 ? b3 : 0x7fu) << 24);
}
__device__ __forceinline__ void pack_scales(const TileArgs& args, int row0, int col0, int kb, int lane, const RawScales& raw, uint32_t (&a)[4], uint32_t (&b)[2][4]) {
    const int live = args.scale_blocks - kb * 4;
#pragma unroll
    for (int g = 0; g < 4; ++g) {
        a[g] = args.sfa_words ? raw.a[g] : pack_word(raw.a[g], raw.a_more[g][0], raw.a_more[g][1], raw.a_more[g][2], live);
        if (row0 + g * 32 + lane >= args.m_total) a[g] = 0x7f7f7f7fu;
    }
#pragma unroll
    for (int c = 0; c < 2; ++c)
#pragma unroll
        for (int g = 0; g < 4; ++g) {
            b[c][g] = pack_word(raw.b[c][g][0], raw.b[c][g][1], raw.b[c][g][2], raw.b[c][g][3], live);
            if (col0 + c * 128 + g * 32 + lane >= args.n_total) b[c][g] = 0x7f7f7f7fu;
        }
}

// A work item's tile, first column and width.
struct Item {
    int m_tile, col0, width;
};
__device__ __forceinline__ Item item_at(const TileArgs& args, int item) {
    int tile = item, half = 0;
    Item out;
    out.width = args.bn;
    if (item >= args.whole_items) {
        tile = args.whole_items + ((item - args.whole_items) >> 1);
        half = (item - args.whole_items) & 1;
        out.width = args.bn >> 1;
    }
    const int n_tile = tile / args.m_tiles;
    out.m_tile = tile - n_tile * args.m_tiles;
    out.col0 = n_tile * args.bn + half * out.width;
    return out;
}

template <int KIND, int CG>
__global__ void __launch_bounds__(thread_count<KIND>(), 1)
umma_matmul_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, const __grid_constant__ CUtensorMap map_c,
                   const __grid_constant__ TileArgs args) {
    constexpr int kCode = KIND == kSixteen ? 0 : (KIND == kCodes || KIND == kCodesSummed ? 20 : (KIND == kScaled ? 40 : (kHasPieces<KIND> ? 60 : (KIND == kSummed ? 80 : 90))));
    constexpr bool kSixteenBits = KIND == kSixteen || kHasPieces<KIND> || KIND == kSummed;
    constexpr int kPieceCount = kHasPieces<KIND> ? 3 : 1;
    constexpr bool kCodesOnly = KIND == kCodes || KIND == kCodesSummed;
    constexpr int kBatch = KIND == kSummed ? 16 : 32;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t* generic_base = smem_raw + (smem_base - smem_u32(smem_raw));
    const uint32_t bar_base = smem_base + args.barrier_offset;
    auto full_bar = [&](int s) { return bar_base + 8u * s; };
    auto empty_bar = [&](int s) { return bar_base + 8u * (kMaxStages + s); };
    auto acc_full = [&](int a) { return bar_base + 8u * (2 * kMaxStages + a); };
    auto acc_empty = [&](int a) { return bar_base + 8u * (2 * kMaxStages + 2 + a); };
    const uint32_t overlap_free = bar_base + 8u * (2 * kMaxStages + 4);
    const uint32_t tmem_slot = bar_base + 8u * (2 * kMaxStages + 5);
    volatile uint32_t* tmem_slot_ptr = reinterpret_cast<volatile uint32_t*>(generic_base + args.barrier_offset + 8 * (2 * kMaxStages + 5));

    const int warp = uniform_warp_index(), lane = threadIdx.x & 31;
    const bool leader = elect_one();
    const bool split = CG == 1 && args.splits > 1;
    const int rank = CG == 2 || split ? static_cast<int>(cluster_rank()) : 0;
    const int group = CG == 2 ? 2 : args.splits;            // CTAs that share a tile
    const int first_item = static_cast<int>(blockIdx.x) / group, item_step = static_cast<int>(gridDim.x) / group;
    const int kb_begin = split ? rank * args.k_per_split : 0;
    const int kb_end = split ? min(args.k_blocks, kb_begin + args.k_per_split) : args.k_blocks;
    const int bn = args.bn;
    const bool overlapped = KIND == kScaled && args.acc_stride < bn;

    if (threadIdx.x == 0) {
        prefetch_tensormap(&map_a);
        prefetch_tensormap(&map_b);
        if (args.tma_store) prefetch_tensormap(&map_c);
    }
    if (warp == 0 && leader) {
        for (int s = 0; s < args.stages; ++s) {
            mbar_init(full_bar(s), kHasScales<KIND> ? 1 + CG : 1);   // the byte count, and the slot's scale warp of each CTA
            mbar_init(empty_bar(s), 1);
        }
        for (int a = 0; a < 2; ++a) {
            mbar_init(acc_full(a), 1);
            mbar_init(acc_empty(a), 8 * CG);
        }
        mbar_init(overlap_free, 4 * CG);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        alloc_columns<CG>(tmem_slot);
        tc_fence_before();
    }
    __syncthreads();
    if (CG == 2) cluster_sync_all();   // both CTAs' barriers exist before either touches the other's
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot_ptr;
    chain_wait();
    chain_release();
    bool settled = !kInBlocks<KIND>;   // (CG = 2, a warp's own answer; the epilogue warps know it for the scale warps too) CTA 0 has waited for every arrival that this CTA's threads sent it

    if (warp == 0) {
        // ---- loader: this CTA's rows of A and share of B; with CG = 2 the bytes are counted on CTA 0's barrier ----
        const uint32_t counted_on = CG == 2 ? address_in(bar_base, 0) : bar_base;
        int stage = 0;
        uint32_t phase = 1;
        bool ok = true;
        for (int i = first_item; i < args.items && ok; i += item_step) {
            const Item item = item_at(args, i);
            const int columns = item.width / CG, boxes = (columns + args.b_box_columns - 1) / args.b_box_columns;
            const int row0 = (item.m_tile * CG + (CG == 2 ? rank : 0)) * kRows, col0 = item.col0 + (CG == 2 ? rank * columns : 0);
            for (int kb = kb_begin; kb < kb_end; ++kb) {
                ok = mbar_wait_warp<true>(empty_bar(stage), phase, 501 + kCode);
                if (!ok) break;
                if (leader) {
                    const uint32_t bar = counted_on + 8u * stage;
                    constexpr int kPerRow = kSixteenBits ? 64 : 128;   // elements of K per block
                    if (CG == 1 || rank == 0) mbar_expect_tx(full_bar(stage), CG * kPieceCount * (args.a_bytes + boxes * args.b_box_bytes));
                    // (pieces: the rows of one follow those of the one before in the same map. A tile that hangs over the end of a
                    // piece reads the next one's first rows, for rows and columns of C that are not stored; past the end of K it is A that holds zeros.)
#pragma unroll
                    for (int piece = 0; piece < kPieceCount; ++piece) {
                        const uint32_t a_dst = smem_base + stage * args.stage_bytes + piece * args.a_bytes;
                        const uint32_t b_dst = smem_base + stage * args.stage_bytes + kPieceCount * args.a_bytes + piece * (bn / CG) * kRowBytes;
                        load_tile<CG>(a_dst, &map_a, kb * kPerRow, row0 + piece * args.a_piece_rows, bar);
                        for (int j = 0; j < boxes; ++j) {
                            if (args.b_mn_major) load_tile<CG>(b_dst + j * args.b_box_bytes, &map_b, col0 + j * args.b_box_columns, kb * kPerRow + piece * args.b_piece_rows, bar);
                            else load_tile<CG>(b_dst + j * args.b_box_bytes, &map_b, kb * kPerRow, col0 + j * args.b_box_columns + piece * args.b_piece_rows, bar);
                        }
                    }
                }
                __syncwarp();
                if (++stage == args.stages) { stage = 0; phase ^= 1; }
            }
        }
    } else if (warp == 1) {
        // ---- issuing warp (of CTA 0 in a pair) ----
        if (CG == 1 || rank == 0) {
            const uint32_t tmem_u = __shfl_sync(0xffffffffu, tmem_base, 0);
            const uint32_t b_lbo = args.b_mn_major ? (kSixteenBits ? 64 * kRowBytes : 128 * kRowBytes) : 16;
            const uint32_t b_step = args.b_mn_major ? (kSixteenBits ? 2048u >> 4 : 4096u >> 4) : 32u >> 4;
            int stage = 0, local = 0;
            uint32_t phase = 0;
            bool ok = true;
            for (int i = first_item; i < args.items; i += item_step, local += kInBlocks<KIND> ? 0 : 1) {
                const int width = item_at(args, i).width, acc = local & args.acc_shift, use = local >> args.acc_shift;
                const uint32_t idesc_wide = args.idesc | (static_cast<uint32_t>(width >> 3) << 17);
                if (!kInBlocks<KIND> && ok) ok = wait_warp<CG == 2>(acc_empty(acc), (use & 1) ^ 1, 502 + kCode);
                // (where the accumulators overlap, the other one's shared columns must have been read out too)
                if (overlapped && ok && local > 0) ok = mbar_wait_warp<true>(overlap_free, (local - 1) & 1, 507 + kCode);
                tc_fence_after();
                uint32_t d = tmem_u + acc * args.acc_stride;
                int in_sum = 0;
                for (int kb = kb_begin; kb < kb_end && ok; ++kb) {
                    const int block_acc = local & args.acc_shift;
                    if (kInBlocks<KIND> && in_sum == 0) {   // (an accumulator per blocks_per_sum blocks)
                        ok = wait_warp<CG == 2>(acc_empty(block_acc), ((local >> args.acc_shift) & 1) ^ 1, 502 + kCode);
                        if (!ok) break;
                        tc_fence_after();
                        d = tmem_u + block_acc * args.acc_stride;
                    }
                    ok = mbar_wait_warp<true>(full_bar(stage), phase, 503 + kCode);
                    if (!ok) break;   // (operands by TMA, scales by generic stores + fence.proxy.async: no tcgen05 fence needed)
                    if (leader) {
                        const uint32_t a_src = smem_base + stage * args.stage_bytes, b_src = a_src + kPieceCount * args.a_bytes;   // (with few rows the products read on into B: rows of C nobody stores)
                        const uint32_t a_lo = smem_desc_lo(a_src, 16), b_lo = smem_desc_lo(b_src, b_lbo);
                        uint32_t sf = 0;
                        if constexpr (kHasScales<KIND>) {
                            const uint32_t scales = b_src + bn / CG * kRowBytes;
                            sf = tmem_u + args.scale_columns + (stage & 1) * 16;   // A's at +0..3, B's at +4..11
                            copy_scales<CG>(sf, scales);
                            copy_scales<CG>(sf + 4, scales + 512);
                            if (width > 128) copy_scales<CG>(sf + 8, scales + 1024);
                        }
                        if constexpr (kHasPieces<KIND>) {
                            // middle*middle, low*high, high*low, middle*high, high*middle meet in an accumulator of their own: the tensor
                            // cores cut off what a sum does not hold, and beside high*high (2^8 times larger) every one of them would lose as much as it does.
                            constexpr int piece_a[6] = {1, 2, 0, 1, 0, 0}, piece_b[6] = {1, 0, 2, 0, 1, 0};
                            const uint32_t a_piece = static_cast<uint32_t>(args.a_bytes) >> 4, b_piece = static_cast<uint32_t>(bn / CG * kRowBytes) >> 4;
#pragma unroll
                            for (int pair = 0; pair < 6; ++pair)
#pragma unroll
                                for (int j = 0; j < 4; ++j)
                                    product<KIND, CG>(pair == 5 ? d : d + bn, desc_words(a_lo + piece_a[pair] * a_piece + ((j * 32) >> 4), smem_desc_hi(1024)),
                                                      desc_words(b_lo + piece_b[pair] * b_piece + j * b_step, smem_desc_hi(1024)), idesc_wide,
                                                      (kInBlocks<KIND> ? in_sum != 0 : kb != kb_begin) || j != 0 || (pair != 0 && pair != 5) ? 1u : 0u, 0u, 0u);
                        } else
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            uint32_t idesc = idesc_wide;
                            if constexpr (kHasScales<KIND>) idesc |= (static_cast<uint32_t>(j) << 29) | (static_cast<uint32_t>(j) << 4);   // the K block's byte of the scale words
                            product<KIND, CG>(d, desc_words(a_lo + ((j * 32) >> 4), smem_desc_hi(1024)), desc_words(b_lo + j * b_step, smem_desc_hi(1024)), idesc,
                                              (kInBlocks<KIND> ? in_sum != 0 : kb != kb_begin) || j != 0 ? 1u : 0u, sf, sf + 4);
                        }
                        commit_to_all<CG>(empty_bar(stage));
                        if (kInBlocks<KIND> && (in_sum + 1 == args.blocks_per_sum || kb + 1 == kb_end)) commit_to_all<CG>(acc_full(block_acc));
                    }
                    if (kInBlocks<KIND> && (++in_sum == args.blocks_per_sum || kb + 1 == kb_end)) {
                        in_sum = 0;
                        ++local;
                    }
                    __syncwarp();
                    if (++stage == args.stages) { stage = 0; phase ^= 1; }
                }
                if (!kInBlocks<KIND> && leader) commit_to_all<CG>(acc_full(acc));   // arrives even after a failed wait, so that no epilogue hangs
                __syncwarp();
            }
        }
    } else if (warp >= 4 && warp < 12) {
        // ---- epilogue: this CTA's 128 rows, group g the boxes g, g + 2, ... of 128 bytes of C each ----
        const int quadrant = warp & 3, g = (warp - 4) >> 2, row = quadrant * 32 + lane;
        const uint32_t lane_base = static_cast<uint32_t>(quadrant * 32) << 16;
        bool ok = true;
        float sums[2][32];   // (kInRegisters)
        if (split) {
            // park the f32 partial tile where the operands were: rows of bn floats, 16-byte units swizzled by the row
            if constexpr (kInRegisters<KIND>) {
                int local = 0;
                sum_blocks<CG>(sums, tmem_base + lane_base, args.acc_stride, bn / 32, g, kb_end - kb_begin, local, acc_full(0), acc_empty(0), lane, ok);
            } else if constexpr (kInPlace<KIND>) {
                int local = 0;
                sum_blocks_in_place<KIND, CG>(args, tmem_base + lane_base, bn / 32, g, kb_end - kb_begin, local, acc_full(0), acc_empty(0), lane, ok);
            } else {
                ok = mbar_wait<true>(acc_full(0), 0, 504 + kCode);
                tc_fence_after();
            }
            uint8_t* parked = generic_base + row * bn * 4;
            for (int c = g; c < bn / 32; c += 2) {
                uint32_t raw[32];
                if constexpr (kInRegisters<KIND>) {
#pragma unroll
                    for (int e = 0; e < 32; ++e) {
                        raw[e] = __float_as_uint(sums[0][e]);
                        sums[0][e] = sums[1][e];
                    }
                } else {
                    tmem_load_32(tmem_base + lane_base + (kInPlace<KIND> ? args.sums_column : 0) + c * 32, raw);
                    tmem_load_wait();
                }
                if constexpr (KIND == kPieces) add_small_products(tmem_base + lane_base + bn + c * 32, raw);
#pragma unroll
                for (int j = 0; j < 8; ++j)
                    *reinterpret_cast<uint4*>(parked + ((c * 8 + (j ^ (row & 7))) << 4)) = make_uint4(raw[4 * j], raw[4 * j + 1], raw[4 * j + 2], raw[4 * j + 3]);
            }
            tc_fence_before();
        } else {
            const uint32_t leader_bars = CG == 2 ? address_in(bar_base, 0) : bar_base;
            const int staging0 = args.staging_offset + g * args.staging_boxes * kStageBox;
            const int box_columns = !args.tma_store || args.out_dtype == DFGPU_F32 ? 32 : (args.out_dtype == DFGPU_E4M3 ? 128 : 64);
            Scalars scalars = load_scalars<kCodesOnly>(args);
            int stored = 0;   // boxes this group has sent off
            int local = 0, status = 0;
            const bool ahead = (KIND == kSixteen || KIND == kPieces) && args.step_count > 0 && args.step_kind[0] != kStepRelu && args.step_dtype[0] != DFGPU_F32;
            uint32_t first_operand[16];
            for (int i = first_item; i < args.items; i += item_step, local += kInBlocks<KIND> ? 0 : 1) {
                const int acc = local & args.acc_shift, use = local >> args.acc_shift;
                const Item item = item_at(args, i);
                const int row0 = (item.m_tile * CG + (CG == 2 ? rank : 0)) * kRows, out_row = row0 + row;
                const bool row_live = out_row < args.m_total;
                // (the first operand of a part is loaded under the part before, of an item's first part under its products: waited for
                // in its place it cost 700 clocks of every part's 2300)
                if (ahead) load_ahead(args, first_operand, out_row, item.col0 + g * box_columns, row_live);
                if constexpr (kInRegisters<KIND>) {
                    sum_blocks<CG>(sums, tmem_base + lane_base, args.acc_stride, item.width / 32, g, kb_end - kb_begin, local, acc_full(0), leader_bars + (acc_empty(0) - bar_base), lane, ok);
                } else if constexpr (kInPlace<KIND>) {
                    sum_blocks_in_place<KIND, CG>(args, tmem_base + lane_base, item.width / 32, g, kb_end - kb_begin, local, acc_full(0), leader_bars + (acc_empty(0) - bar_base), lane, ok);
                } else {
                    if (ok) ok = mbar_wait<true>(acc_full(acc), use & 1, 505 + kCode);
                    tc_fence_after();
                }
                status = ask_status();
                const uint32_t columns = tmem_base + lane_base + (kInPlace<KIND> ? args.sums_column : acc * args.acc_stride);
                const int boxes = item.width / box_columns;
                for (int b = g; b < boxes; b += 2) {
                    // overlapping accumulators: the first one is read from its end, the second from its start
                    const int box = overlapped && acc == 0 ? boxes - 2 + 2 * g - b : b;
                    const int col0 = item.col0 + box * box_columns;
                    const int staging = staging0 + (args.staging_boxes == 2 ? (stored & 1) * kStageBox : 0);
                    if (args.tma_store && stored >= args.staging_boxes) {
                        if (row == 0) {
                            if (args.staging_boxes == 2) tma_store_wait_read<1>();
                            else tma_store_wait_read<0>();
                        }
                        epilogue_barrier(1 + g);
                    }
                    for (int part = 0; part < box_columns / 32; ++part) {
                        uint32_t raw[32];
                        if constexpr (kInRegisters<KIND>) {   // (f32 C: boxes of 32 columns)
#pragma unroll
                            for (int e = 0; e < 32; ++e) {
                                raw[e] = __float_as_uint(sums[0][e]);
                                sums[0][e] = sums[1][e];   // (the group's second box is next)
                            }
                        } else {
                            tmem_load_32(columns + box * box_columns + part * 32, raw);
                            tmem_load_wait();
                        }
                        if constexpr (KIND == kPieces) add_small_products(columns + bn + box * box_columns + part * 32, raw);
                        if (overlapped && b == g && g != acc && part == box_columns / 32 - 1) {   // the shared columns are in registers
                            tc_fence_before();
                            __syncwarp();
                            if (lane == 0) {
                                if (CG == 2 && i + item_step < args.items) mbar_arrive_cluster(leader_bars + (overlap_free - bar_base));   // (one that nobody waits for could come when CTA 0 has left)
                                if (CG == 1) mbar_arrive(overlap_free);
                            }
                        }
                        float v[32];
#pragma unroll
                        for (int e = 0; e < 32; ++e) v[e] = __uint_as_float(raw[e]);
                        const int col = col0 + part * 32;
                        if (ahead) {
                            uint32_t operand[16];
#pragma unroll
                            for (int e = 0; e < 16; ++e) operand[e] = first_operand[e];
                            const bool same_box = part + 1 < box_columns / 32;
                            if (same_box || b + 2 < boxes) load_ahead(args, first_operand, out_row, same_box ? col + 32 : item.col0 + (b + 2) * box_columns, row_live);
                            apply_steps<kCodesOnly, kBatch, 32>(args, v, out_row, col, row_live, scalars, &operand);
                        } else {
                            apply_steps<kCodesOnly, kBatch, 32>(args, v, out_row, col, row_live, scalars);
                        }
                        if (args.tma_store) {
                            uint8_t* target = generic_base + staging + row * 128;
                            if (kInRegisters<KIND> || KIND == kScaledSummed || args.out_dtype == DFGPU_F32) {   // (those have f32 results only)
#pragma unroll
                                for (int j = 0; j < 8; ++j)
                                    *reinterpret_cast<float4*>(target + ((j ^ (row & 7)) << 4)) = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
                            } else if (args.out_dtype == DFGPU_E4M3) {
#pragma unroll
                                for (int j = 0; j < 2; ++j)
                                    *reinterpret_cast<uint4*>(target + (((part * 2 + j) ^ (row & 7)) << 4)) =
                                        make_uint4(encode_four_e4m3(v + 16 * j), encode_four_e4m3(v + 16 * j + 4), encode_four_e4m3(v + 16 * j + 8), encode_four_e4m3(v + 16 * j + 12));
                            } else {
                                auto put = [&](int dtype) {   // (one branch for all)
#pragma unroll
                                    for (int j = 0; j < 4; ++j)
                                        *reinterpret_cast<uint4*>(target + (((part * 4 + j) ^ (row & 7)) << 4)) =
                                            make_uint4(narrow_pair(v[8 * j], v[8 * j + 1], dtype), narrow_pair(v[8 * j + 2], v[8 * j + 3], dtype),
                                                       narrow_pair(v[8 * j + 4], v[8 * j + 5], dtype), narrow_pair(v[8 * j + 6], v[8 * j + 7], dtype));
                                };
                                if (args.out_dtype == DFGPU_BF16) put(DFGPU_BF16);
                                else put(DFGPU_F16);
                            }
                        } else if (row_live && healthy_now(ok, status)) {
                            const int64_t at = out_row * args.out_ld + col;
#pragma unroll
                            for (int e = 0; e < 32; ++e)
                                if (col + e < args.n_total) store_from_f32(args.out, args.out_dtype, at + e, v[e]);
                        }
                    }
                    if (args.tma_store) {
                        fence_async_shared();
                        epilogue_barrier(1 + g);
                        if (row == 0) {
                            if (healthy_now(ok, status) && row0 < args.m_total && col0 < args.n_total) tma_store_2d(&map_c, smem_base + staging, col0, row0);
                            tma_store_commit();
                        }
                        ++stored;
                    }
                }
                tc_fence_before();
                __syncwarp();
                if (!kInBlocks<KIND> && lane == 0) {
                    if (CG == 2 && i + item_step * (args.acc_shift + 1) < args.items) mbar_arrive_cluster(leader_bars + 8u * (2 * kMaxStages + 2 + acc));
                    if (CG == 1) mbar_arrive(acc_empty(acc));
                }
            }
            if (args.tma_store && row == 0) tma_store_wait_all();
            if (CG == 2) settled = __all_sync(0xffffffffu, settled && healthy_now(ok, status)) != 0;
            __syncwarp();
            fold_amax<kCodesOnly>(args, scalars, lane, ok);
        }
    } else if (kHasScales<KIND>) {
        // ---- scale loaders: warp i of the six owns the slots i and i + 6 ----
        // (A slot has ONE owner: the parity of its barrier tells apart two rounds, not three, so a warp that came by a slot
        // only every other round could fill it before its last round was read.)
        const int me = warp < 4 ? warp - 2 : warp - 10;
        constexpr int kScaleWarps = 6;   // (no fewer than the slots of a 256-column ring: a warp with two slots set the pace)
        // position in the list of (work item, K block) pairs this CTA walks, `stage` the slot of the pair
        int at = first_item, kb = kb_begin, stage = 0;
        uint32_t phase = 1;
        auto advance = [&] {
            if (++stage == args.stages) { stage = 0; phase ^= 1; }
            if (++kb == kb_end) { kb = kb_begin; at += item_step; }
        };
        auto seek = [&] {   // the next pair in one of this warp's slots
            while (at < args.items && stage % kScaleWarps != me) advance();
            return at < args.items;
        };
        RawScales raw;
        Item item = item_at(args, at);
        auto load = [&] {
            item = item_at(args, at);
            load_scales(args, (item.m_tile * CG + (CG == 2 ? rank : 0)) * kRows, item.col0, kb, lane, raw);
        };
        bool more = kb_begin < kb_end && seek();
        if (more) load();
        while (more) {
            const int slot = stage;
            const uint32_t slot_phase = phase;
            uint32_t a_words[4], b_words[2][4];
            pack_scales(args, (item.m_tile * CG + (CG == 2 ? rank : 0)) * kRows, item.col0, kb, lane, raw, a_words, b_words);
            advance();
            more = seek();
            if (more) load();
            if (!mbar_wait_warp<true>(empty_bar(slot), slot_phase, 506 + kCode)) break;
            uint8_t* scales = generic_base + slot * args.stage_bytes + args.a_bytes + bn / CG * kRowBytes + lane * 16;
            *reinterpret_cast<uint4*>(scales) = make_uint4(a_words[0], a_words[1], a_words[2], a_words[3]);
            *reinterpret_cast<uint4*>(scales + 512) = make_uint4(b_words[0][0], b_words[0][1], b_words[0][2], b_words[0][3]);
            if (bn > 128) *reinterpret_cast<uint4*>(scales + 1024) = make_uint4(b_words[1][0], b_words[1][1], b_words[1][2], b_words[1][3]);
            fence_async_shared();
            __syncwarp();
            if (leader) {
                // CTA 0's products read both CTAs' scales, each from its CTA's own shared memory and by the asynchronous proxy, to which
                // fence.proxy.async has made every lane's stores visible before the warp met: no thread of CTA 0 reads them, so there is
                // nothing that a release to the cluster would order besides (it waits for its round trip, 89 -> 100 us at 4096^3)
                if (CG == 2) mbar_arrive_cluster(address_in(full_bar(slot), 0));
                else mbar_arrive(full_bar(slot));
            }
        }
    }

    if (split) {
        // ---- the cluster's partial tiles: every CTA adds its share of the live rows over all ranks, in rank order ----
        // (Latencies one behind the other: what does not need the other CTAs, places and the first fused operand, is fetched while they
        // arrive, and the others may leave once this CTA has their partial sums, which its own stores need not be done for, as a release would wait for:
        // with bias and ReLU 100 x 544 x 1008 f16 6.13 -> 4.82 us, 128 x 4096 x 4096 bf16 out of HBM 13.6 -> 11.7, in L2 11.6 -> 10.0; FP8 117 x 1040 x 416 7.20 -> 6.06.)
        cluster_arrive();   // (all threads: this CTA's partial tile is in place)
        const Item item = item_at(args, first_item);
        const int row0 = item.m_tile * kRows, live_rows = min(kRows, args.m_total - row0);
        const int share = (live_rows + args.splits - 1) / args.splits, begin = rank * share, end = min(live_rows, begin + share);
        const int quad_bits = 31 - __clz(bn >> 2), count = max(0, end - begin) << quad_bits;   // (bn is 64 or 128)
        Scalars scalars = load_scalars<kCodesOnly>(args);
        const bool ahead = !kCodesOnly && args.step_count > 0 && args.step_kind[0] != kStepRelu && args.step_dtype[0] != DFGPU_F32;
        uint32_t operand[2] = {};
        auto row_of = [&](int i) { return begin + (i >> quad_bits); };
        auto column_of = [&](int i) { return item.col0 + (i & ((1 << quad_bits) - 1)) * 4; };
        auto fetch = [&](int i) {
            const int col = column_of(i);
            if (ahead && i < count && col < args.n_total)
                load_words<4>(operand, static_cast<const uint16_t*>(args.step_data[0]) + (args.step_kind[0] == kStepBias ? 0 : (row0 + row_of(i)) * args.step_ld[0]) + col, args.n_total - col,
                              args.step_vector[0] != 0);
        };
        fetch(static_cast<int>(threadIdx.x));
        cluster_wait();
        const int status = ask_status();
        bool rare = false;
        for (int i = threadIdx.x; i < count; i += static_cast<int>(blockDim.x)) {
            const int row = row_of(i), unit = i & ((1 << quad_bits) - 1), col = column_of(i);
            if (col >= args.n_total) continue;   // (and so are this thread's further columns: its unit stays)
            const uint32_t at = smem_base + row * bn * 4 + (((unit & ~7) | ((unit ^ row) & 7)) << 4);
            constexpr int kMost = 8;
            float4 part[kMost];
#pragma unroll
            for (int z = 0; z < kMost; ++z)   // every load in flight before the first sum
                if (z < args.splits) part[z] = load_from_rank(address_in(at, z));
            float v[4] = {part[0].x, part[0].y, part[0].z, part[0].w};
#pragma unroll
            for (int z = 1; z < kMost; ++z) {
                if (z >= args.splits) break;
                v[0] = __fadd_rn(v[0], part[z].x);
                v[1] = __fadd_rn(v[1], part[z].y);
                v[2] = __fadd_rn(v[2], part[z].z);
                v[3] = __fadd_rn(v[3], part[z].w);
            }
            rare = rare || __float_as_uint(v[0]) == kRareSum;
            if (ahead) apply_steps<kCodesOnly, 4, 4>(args, v, row0 + row, col, true, scalars, &operand);
            else apply_steps<kCodesOnly, 4, 4>(args, v, row0 + row, col, true, scalars);
            if (healthy_now(true, status)) store_four(args, v, row0 + row, col);
            fetch(i + static_cast<int>(blockDim.x));
        }
        __syncwarp();
        cluster_arrive_behind_loads(rare);
        fold_amax<kCodesOnly>(args, scalars, lane, healthy_now(true, status));
        cluster_wait();   // no CTA leaves while another still reads its partial tile
    }
    tc_fence_before();
    const bool all_settled = CG == 2 && kHasScales<KIND> ? __syncthreads_and(settled) != 0 : (__syncthreads(), settled);
    if (CG == 2) {   // ... or may still signal its barriers or read its operands
        // (The stores of C go to nobody here: a release, which waits until they are done, is for the arrivals at CTA 0's barriers alone, and
        // those that it waits for have come before the accumulators that the epilogue waited for. Where a wait gave up, the scale warps' last arrivals may have been
        // waited for by nobody, and they release too. FP8 777 x 4096 x 3072 with the shorter waits of its epilogue 15.0 -> 14.5 us, bf16 2048^3 15.0 -> 14.5.)
        if (all_settled) cluster_arrive_relaxed();
        else cluster_arrive();
        cluster_wait();
    }
    if (warp == 1) {
        tc_fence_after();
        free_columns<CG>(tmem_base);
    }
}

// ---- host --------------------------------------------------------------------------------------------------

bool on16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

int encode_map(CUtensorMap* map, CUtensorMapDataType type, const void* base, int64_t inner, int64_t outer, int64_t stride_bytes, uint32_t box_inner,
               uint32_t box_outer, const char* what) {
    EncodeTiled encode = encode_tiled();
    if (!encode) return fail(kExecutionFailed, "%s: cuTensorMapEncodeTiled is unavailable", what);
    cuuint64_t dims[2] = {static_cast<cuuint64_t>(inner), static_cast<cuuint64_t>(outer)}, strides[1] = {static_cast<cuuint64_t>(stride_bytes)};
    cuuint32_t box[2] = {box_inner, box_outer}, element_strides[2] = {1, 1};
    CUresult result = encode(map, type, 2, const_cast<void*>(base), dims, strides, box, element_strides, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                             CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (result != CUDA_SUCCESS) return fail(kExecutionFailed, "%s: tensor map encode failed (CUresult %d)", what, static_cast<int>(result));
    return kOk;
}

bool row_ok(int64_t ld, int64_t extent, int bytes) { return ld >= extent && (ld * bytes) % 16 == 0 && ld * bytes < (1ll << 40); }

// A and B must be readable by TMA: contiguous rows that start on 16-byte boundaries (a single row has no stride to mind).
bool describe(const dfgpu_tensor& a, const dfgpu_tensor& b, const dfgpu_tensor& c, int kind, Problem& p) {
    const int rank = c.rank;
    if (rank < 2 || a.rank != rank || b.rank != rank) return false;
    for (int i = 0; i < rank - 2; ++i)
        if (a.dim[i] != 1 || b.dim[i] != 1 || c.dim[i] != 1) return false;
    p.kind = kind;
    p.M = c.dim[rank - 2];
    p.N = c.dim[rank - 1];
    p.K = a.dim[rank - 1];
    if (a.dim[rank - 2] != p.M || b.dim[rank - 2] != p.K || b.dim[rank - 1] != p.N) return false;
    if (p.M < 1 || p.N < 1 || p.K < 1 || p.M > (1ll << 28) || p.N > (1ll << 28) || p.K > (1ll << 28)) return false;
    p.in_bytes = kind == kSixteen || kind == kSummed ? 2 : 1;
    p.a_rows = p.M;
    p.out_dtype = c.dtype;
    p.out_bytes = dtype_bytes(c.dtype);
    p.a_ld = a.stride[rank - 2];
    if (p.M == 1) p.a_ld = (p.K * p.in_bytes + 15) / 16 * 16 / p.in_bytes;
    if (a.stride[rank - 1] != 1 || !row_ok(p.a_ld, p.K, p.in_bytes)) return false;
    const bool k_major = b.stride[rank - 2] == 1 && row_ok(b.stride[rank - 1], p.K, p.in_bytes);
    p.b_mn_major = !k_major;
    p.b_ld = k_major ? b.stride[rank - 1] : b.stride[rank - 2];
    if (!k_major && (b.stride[rank - 1] != 1 || !row_ok(p.b_ld, p.N, p.in_bytes))) return false;
    p.b_rows = k_major ? p.N : p.K;
    p.c_ld = c.stride[rank - 2];
    return c.stride[rank - 1] == 1 && p.c_ld >= p.N;
}

template <int KIND, int CG>
int launch_kernel(const CUtensorMap& map_a, const CUtensorMap& map_b, const CUtensorMap& map_c, const TileArgs& args, int grid, int dynamic, cudaStream_t stream, const char* what) {
    // (the most that any shape takes, and not this one's need: the attribute belongs to the function, and a launch of a larger
    // shape between this call and the next, on another thread or repeated without it, would be refused)
    constexpr int kMostDynamic = kSmemBudget + 1024;
    if (dynamic > kMostDynamic) return fail(kExecutionFailed, "%s: %d bytes of shared memory", what, dynamic);
    cudaError_t error = cudaFuncSetAttribute(umma_matmul_kernel<KIND, CG>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMostDynamic);
    if (error != cudaSuccess) return fail(kExecutionFailed, "%s: cannot reserve %d bytes of shared memory: %s", what, kMostDynamic, cudaGetErrorString(error));
    const unsigned cluster = CG == 2 ? 2u : (args.splits > 1 ? static_cast<unsigned>(args.splits) : 0u);
    error = launch_chained_cluster(umma_matmul_kernel<KIND, CG>, dim3(static_cast<unsigned>(grid)), dim3(thread_count<KIND>()), cluster, static_cast<size_t>(dynamic), stream,
                                   map_a, map_b, map_c, args);
    if (error != cudaSuccess) return fail(kExecutionFailed, "%s: launch failed: %s", what, cudaGetErrorString(error));
    return check_launch(what);
}

// Everything but the epilogue's operands and the operand formats, which the callers have put into `args`.
int launch_problem(Problem p, TileArgs& args, const void* a, const void* b, void* c, cudaStream_t stream, const char* what) {
    p.direct_stores = !on16(c) || (p.c_ld * p.out_bytes) % 16 != 0 || p.out_dtype == DFGPU_E5M2;
    int operands = 0;   // full ADD operands that are not loaded ahead
    for (int s = 0; s < args.step_count; ++s) operands += args.step_kind[s] == kStepFull && (s > 0 || args.step_dtype[s] == DFGPU_F32 || p.kind != kSixteen) ? 1 : 0;
    const Shape shape = choose_shape(p, operands);
    const int chunk = sixteen_bits(p) ? 64 : 128;
    args.m_total = static_cast<int>(p.M);
    args.n_total = static_cast<int>(p.N);
    args.bn = shape.bn;
    args.m_tiles = static_cast<int>((p.M + kRows * shape.cg - 1) / (kRows * shape.cg));
    args.k_blocks = static_cast<int>((p.K * p.in_bytes + kRowBytes - 1) / kRowBytes);
    args.splits = shape.splits;
    args.k_per_split = shape.k_per_split;
    args.b_mn_major = p.b_mn_major ? 1 : 0;
    const int columns = shape.bn / shape.cg;   // of B per CTA
    args.b_box_columns = p.b_mn_major ? chunk : (shape.halved > 0 ? columns / 2 : columns);
    args.whole_items = static_cast<int>(shape.tiles - shape.halved);
    args.items = static_cast<int>(shape.tiles + shape.halved);
    args.b_box_bytes = (p.b_mn_major ? kRowBytes / p.in_bytes : args.b_box_columns) * kRowBytes;   // N-major: one row of 128 bytes per element of K
    const int a_rows = rows_of_a(p, shape.cg);
    args.a_bytes = a_rows * kRowBytes;
    args.stage_bytes = stage_bytes(p, shape.bn, shape.cg, a_rows);
    args.out = c;
    args.out_ld = p.c_ld;
    args.out_dtype = p.out_dtype;
    args.tma_store = p.direct_stores ? 0 : 1;
    // Tensor memory: two accumulators, and with block scales 32 columns of them at the end. At bn = 256 the accumulators then
    // overlap by 32 columns, which the epilogue reads out first.
    // Pieces: an accumulator is two of bn columns (leading and lower products), so that 192 and 256 columns leave room for one: the
    // epilogue of a tile then runs alone, a few percent of its 6 x K / 64 product steps.
    args.acc_stride = p.kind == kScaled && shape.bn == 256 ? 224 : (has_pieces(p) ? 2 * shape.bn : shape.bn);
    args.acc_shift = (has_pieces(p) && shape.bn > 128) || p.kind == kPiecesSummed ? 0 : 1;
    // (kPiecesSummed: one accumulator of 2 bn columns and the sums behind it; eight blocks each, whose error is half that of f32 additions over
    // 4096 products, so that reading them out costs little)
    args.blocks_per_sum = p.kind == kPiecesSummed ? 8 : 1;
    args.sums_column = (args.acc_shift + 1) * args.acc_stride;
    args.scale_columns = 480;
    const int barriers = (2 * kMaxStages + 6) * 8;
    const int box_columns = kRowBytes / p.out_bytes;
    // (two staging boxes a group where it fills more than one and they leave the ring five stages: a box is otherwise written only when
    // the store before has been read, 400 clocks each. 2048 x 64 x 4096 bf16 with bias and ReLU, with the operands loaded ahead: 12.6 us -> 10.8; MXFP8 4096^3
    // with four stages for five: 0.9 % slower.)
    const bool many_boxes = shape.bn > 2 * box_columns || shape.tiles + shape.halved > sm_count() / shape.cg;
    args.staging_boxes = many_boxes && stages_that_fit(args.stage_bytes, kSmemBudget - 4 * kStageBox - barriers) >= 5 ? 2 : 1;
    const int staging = shape.splits > 1 || !args.tma_store ? 0 : 2 * args.staging_boxes * kStageBox;
    args.stages = stages_that_fit(args.stage_bytes, kSmemBudget - staging - barriers);
    args.staging_offset = ring_bytes(args.stages, args.stage_bytes);   // (a split product parks its 128 x bn partial tile, at most 64 KB, in the ring)
    args.barrier_offset = args.staging_offset + staging;
    const int dynamic = args.barrier_offset + barriers + 1024;
    // instruction descriptor: f32 accumulators (or E8M0 scales), the operand formats the caller has set, B's major, M (N is the item's)
    args.idesc |= (scaled(p) ? 1u << 23 : 1u << 4) | (static_cast<uint32_t>(args.b_mn_major) << 16) |
                  (static_cast<uint32_t>(kRows * shape.cg >> 4) << 24);
    const CUtensorMapDataType in_type = sixteen_bits(p) ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_UINT8;   // (copied, never computed on)
    const uint32_t per_row = kRowBytes / p.in_bytes;
    CUtensorMap map_a, map_b, map_c{};
    int status = encode_map(&map_a, in_type, a, p.K, p.a_rows, p.a_ld * p.in_bytes, per_row, a_rows, what);
    if (!status) {
        if (p.b_mn_major) status = encode_map(&map_b, in_type, b, p.N, p.b_rows, p.b_ld * p.in_bytes, chunk, per_row, what);
        else status = encode_map(&map_b, in_type, b, p.K, p.b_rows, p.b_ld * p.in_bytes, per_row, static_cast<uint32_t>(args.b_box_columns), what);
    }
    if (!status && args.tma_store) {
        const CUtensorMapDataType out_type = p.out_dtype == DFGPU_F32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : (p.out_dtype == DFGPU_E4M3 ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16);
        status = encode_map(&map_c, out_type, c, p.N, p.M, p.c_ld * p.out_bytes, kRowBytes / p.out_bytes, kRows, what);
    }
    if (status) return status;
    const int64_t groups = shape.splits > 1 ? shape.tiles : std::min<int64_t>(shape.tiles, sm_count() / shape.cg);
    const int grid = static_cast<int>(groups * (shape.cg == 2 ? 2 : shape.splits));
    if (p.kind == kSixteen) return shape.cg == 2 ? launch_kernel<kSixteen, 2>(map_a, map_b, map_c, args, grid, dynamic, stream, what) : launch_kernel<kSixteen, 1>(map_a, map_b, map_c, args, grid, dynamic, stream, what);
    if (p.kind == kCodesSummed) return shape.cg == 2 ? launch_kernel<kCodesSummed, 2>(map_a, map_b, map_c, args, grid, dynamic, stream, what) : launch_kernel<kCodesSummed, 1>(map_a, map_b, map_c, args, grid, dynamic, stream, what);
    if (p.kind == kCodes) return shape.cg == 2 ? launch_kernel<kCodes, 2>(map_a, map_b, map_c, args, grid, dynamic, stream, what) : launch_kernel<kCodes, 1>(map_a, map_b, map_c, args, grid, dynamic, stream, what);
    if (p.kind == kSummed) return shape.cg == 2 ? launch_kernel<kSummed, 2>(map_a, map_b, map_c, args, grid, dynamic, stream, what) : launch_kernel<kSummed, 1>(map_a, map_b, map_c, args, grid, dynamic, stream, what);
    if (p.kind == kPiecesSummed) return shape.cg == 2 ? launch_kernel<kPiecesSummed, 2>(map_a, map_b, map_c, args, grid, dynamic, stream, what) : launch_kernel<kPiecesSummed, 1>(map_a, map_b, map_c, args, grid, dynamic, stream, what);
    if (has_pieces(p)) return shape.cg == 2 ? launch_kernel<kPieces, 2>(map_a, map_b, map_c, args, grid, dynamic, stream, what) : launch_kernel<kPieces, 1>(map_a, map_b, map_c, args, grid, dynamic, stream, what);
    if (p.kind == kScaledSummed) return shape.cg == 2 ? launch_kernel<kScaledSummed, 2>(map_a, map_b, map_c, args, grid, dynamic, stream, what) : launch_kernel<kScaledSummed, 1>(map_a, map_b, map_c, args, grid, dynamic, stream, what);
    return shape.cg == 2 ? launch_kernel<kScaled, 2>(map_a, map_b, map_c, args, grid, dynamic, stream, what) : launch_kernel<kScaled, 1>(map_a, map_b, map_c, args, grid, dynamic, stream, what);
}

// The fused steps the kernel applies: ReLU, a per-column ADD operand, a full [M, N] ADD operand with contiguous columns.
bool translate_steps(const dfgpu_matmul_params& p, void* const* tensors, TileArgs* args) {
    if (p.epilogue_count < 0 || p.epilogue_count > kMaxSteps) return false;
    const int rank = p.c.rank;
    if (args) args->step_count = p.epilogue_count;
    for (int i = 0; i < p.epilogue_count; ++i) {
        const dfgpu_epilogue_step& step = p.epilogue[i];
        if (step.op == DFGPU_EPI_RELU) {
            if (args) {
                args->step_kind[i] = kStepRelu;
                args->relu_lower[i] = step.relu_lower;
                args->relu_upper[i] = step.relu_upper;
                args->relu_slope[i] = step.relu_slope;
            }
            continue;
        }
        if (step.op != DFGPU_EPI_ADD || step.operand < 0 || step.operand > 1) return false;
        const dfgpu_tensor& t = p.extra[step.operand];
        if (t.rank < 1 || t.rank > rank || (t.dtype != DFGPU_BF16 && t.dtype != DFGPU_F16 && t.dtype != DFGPU_F32)) return false;
        for (int axis = 0; axis < t.rank - 2; ++axis)
            if (t.dim[axis] != 1) return false;
        if (t.dim[t.rank - 1] != p.c.dim[rank - 1] || (t.stride[t.rank - 1] != 1 && t.dim[t.rank - 1] != 1)) return false;
        const bool per_column = t.rank == 1 || t.dim[t.rank - 2] == 1;
        if (!per_column && t.dim[t.rank - 2] != p.c.dim[rank - 2]) return false;
        if (args) {
            args->step_kind[i] = per_column ? kStepBias : kStepFull;
            args->step_data[i] = tensors[5 + step.operand];
            args->step_dtype[i] = t.dtype;
            args->step_ld[i] = per_column ? 0 : t.stride[t.rank - 2];
            args->step_vector[i] = on16(args->step_data[i]) && (args->step_ld[i] * dtype_bytes(t.dtype)) % 16 == 0 ? 1 : 0;
        }
    }
    return true;
}

// f32 results that are summed block by block: all but those of whole tiles in whole 16-byte units, which always came from one
// accumulator.
bool sums_blocks(const dfgpu_matmul_params& p) {
    const int rank = p.c.rank;
    if (p.c.dtype != DFGPU_F32 || rank < 2 || p.a.rank != rank) return false;
    const bool has_scales = p.a.dtype == DFGPU_E4M3;
    const int64_t M = p.c.dim[rank - 2], N = p.c.dim[rank - 1], K = p.a.dim[rank - 1], tile = has_scales ? 128 : 64;
    if (p.a.dtype == DFGPU_F16 || K % tile != 0 || N % tile != 0 || p.a.stride[rank - 2] % 8 != 0 || p.c.stride[rank - 2] % 8 != 0) return true;
    if (has_scales && (M % 128 != 0 || p.a_scale.stride[rank - 2] % 4 != 0)) return true;
    for (int i = 0; i < std::min<int>(p.epilogue_count, kMaxSteps); ++i) {
        if (p.epilogue[i].op != DFGPU_EPI_ADD || p.epilogue[i].operand < 0 || p.epilogue[i].operand > 1) continue;   // (translate_steps() refuses those)
        const dfgpu_tensor& t = p.extra[p.epilogue[i].operand];
        if (t.rank < 1) continue;
        const bool per_column = t.rank == 1 || t.dim[t.rank - 2] == 1;
        if (t.dtype == DFGPU_F16 || (!has_scales && !per_column && (t.rank != rank || t.stride[rank - 2] != p.c.stride[rank - 2]))) return true;
    }
    return false;
}

bool sixteen_problem(const dfgpu_matmul_params& p, Problem& problem) {
    if (p.a_scale.rank || p.b_scale.rank) return false;
    if ((p.a.dtype != DFGPU_BF16 && p.a.dtype != DFGPU_F16) || p.b.dtype != p.a.dtype) return false;   // (one kind of operand per instruction)
    if (p.c.dtype != DFGPU_BF16 && p.c.dtype != DFGPU_F16 && p.c.dtype != DFGPU_F32) return false;
    // (fewer products in bf16: the CUDA cores' additions are the more exact, 5.4e-8 from 64 bits for 6.3e-8 at 72, 6.0 / 6.4 at 88, 6.6 / 6.6 at 104)
    constexpr int64_t kSummedMinDepth = 104;
    if (p.a.dtype == DFGPU_BF16 && sums_blocks(p) && p.a.dim[p.a.rank - 1] < kSummedMinDepth) return false;
    return translate_steps(p, nullptr, nullptr) && describe(p.a, p.b, p.c, sums_blocks(p) ? kSummed : kSixteen, problem);
}

bool scaled_problem(const dfgpu_matmul_params& p, Problem& problem) {
    if (p.a.dtype != DFGPU_E4M3 || p.b.dtype != DFGPU_E4M3 || p.a_scale.dtype != DFGPU_E8M0 || p.b_scale.dtype != DFGPU_E8M0) return false;
    if (p.c.dtype != DFGPU_BF16 && p.c.dtype != DFGPU_F16 && p.c.dtype != DFGPU_F32) return false;
    const int rank = p.c.rank;
    if (p.a_scale.rank != rank || p.b_scale.rank != rank || !describe(p.a, p.b, p.c, kScaled, problem)) return false;
    if (sums_blocks(p)) problem.kind = kScaledSummed;
    for (int i = 0; i < rank - 2; ++i)
        if (p.a_scale.dim[i] != 1 || p.b_scale.dim[i] != 1) return false;
    if (problem.N <= 64) return false;   // (column scales come in chunks of 128: half of a tile would be empty; dequantized to bf16, N = 64 is a tile)
    // scales: one per 32 elements along K, plain layout
    if (problem.K % 32 != 0 || p.a_block[0] != 1 || p.a_block[1] != 32 || p.b_block[0] != 32 || p.b_block[1] != 1) return false;
    if (p.a_scale.reorder != DFGPU_REORDER_NONE || p.b_scale.reorder != DFGPU_REORDER_NONE) return false;
    if (p.a_scale.dim[rank - 2] != problem.M || p.a_scale.dim[rank - 1] != problem.K / 32 || p.a_scale.stride[rank - 1] != 1) return false;
    if (p.b_scale.dim[rank - 2] != problem.K / 32 || p.b_scale.dim[rank - 1] != problem.N || p.b_scale.stride[rank - 1] != 1) return false;
    return translate_steps(p, nullptr, nullptr);
}

}  // namespace

bool matmul_umma_supported(const dfgpu_matmul_params& p, int kernel) {
    Problem problem;
    return kernel == DFGPU_MATMUL_UMMA_MXF8 ? scaled_problem(p, problem) : (kernel == DFGPU_MATMUL_UMMA_BF16 && sixteen_problem(p, problem));
}

// The pieces' own matrices take the place of A and B: only C and the fused steps have to suit the kernel.
bool matmul_pieces_supported(const dfgpu_matmul_params& p) {
    const int rank = p.c.rank;
    return p.c.stride[rank - 1] == 1 && p.c.stride[rank - 2] >= p.c.dim[rank - 1] && (p.c.dtype == DFGPU_BF16 || p.c.dtype == DFGPU_F16 || p.c.dtype == DFGPU_F32) && translate_steps(p, nullptr, nullptr);
}

int launch_matmul_pieces(const dfgpu_matmul_params& p, const PieceMatmul& pieces, void* const* tensors, cudaStream_t stream) {
    const int rank = p.c.rank;
    Problem problem{};
    problem.M = p.c.dim[rank - 2], problem.N = p.c.dim[rank - 1], problem.K = p.a.dim[rank - 1];
    problem.a_ld = pieces.a_ld, problem.b_ld = pieces.b_ld, problem.c_ld = p.c.stride[rank - 2];
    problem.b_mn_major = pieces.b_n_major;
    // depths beyond the one-launch f32 kernel's, which the CUDA cores summed unless the extents were whole tiles: no further from 64 bits
    problem.kind = problem.K > 4096 && (problem.K % 64 != 0 || problem.N % 64 != 0) ? kPiecesSummed : kPieces;
    problem.in_bytes = 2, problem.out_bytes = dtype_bytes(p.c.dtype), problem.out_dtype = p.c.dtype;
    problem.a_rows = 3 * problem.M;
    problem.b_rows = 3 * (pieces.b_n_major ? problem.K : problem.N);
    TileArgs args{};
    args.idesc = (1u << 7) | (1u << 10);
    args.a_piece_rows = static_cast<int>(problem.M);
    args.b_piece_rows = static_cast<int>(problem.b_rows / 3);
    translate_steps(p, tensors, &args);
    return launch_problem(problem, args, pieces.a, pieces.b, tensors[2], stream, "MATMUL (tcgen05)");
}

int launch_matmul_umma(const dfgpu_matmul_params& p, void* const* tensors, int kernel, cudaStream_t stream) {
    Problem problem;
    TileArgs args{};
    if (!on16(tensors[0]) || !on16(tensors[1])) return fail(kInvalidArgument, "MATMUL: the tcgen05 kernel needs 16-byte aligned A and B");
    if (kernel == DFGPU_MATMUL_UMMA_MXF8) {
        if (!scaled_problem(p, problem)) return fail(kUnsupported, "MATMUL: the tcgen05 kernel does not take these block-scaled operands");
        const int rank = p.c.rank;
        args.sfa = static_cast<const uint8_t*>(tensors[3]);
        args.sfb = static_cast<const uint8_t*>(tensors[4]);
        args.sfa_ld = p.a_scale.stride[rank - 2];
        args.sfb_ld = p.b_scale.stride[rank - 2];
        args.scale_blocks = static_cast<int>(problem.K / 32);
        args.sfa_words = (reinterpret_cast<uintptr_t>(args.sfa) & 3u) == 0 && args.sfa_ld % 4 == 0 && args.scale_blocks % 4 == 0 ? 1 : 0;
    } else {
        if (!sixteen_problem(p, problem)) return fail(kUnsupported, "MATMUL: the tcgen05 kernel does not take these operands");
        if (p.a.dtype == DFGPU_BF16) args.idesc = (1u << 7) | (1u << 10);
    }
    translate_steps(p, tensors, &args);
    return launch_problem(problem, args, tensors[0], tensors[1], tensors[2], stream, "MATMUL (tcgen05)");
}

bool fp8_problem(const dfgpu_matmul_fp8_params& p, Problem& problem) {
    if ((p.a.dtype != DFGPU_E4M3 && p.a.dtype != DFGPU_E5M2) || (p.b.dtype != DFGPU_E4M3 && p.b.dtype != DFGPU_E5M2)) return false;
    if (p.c.dtype != DFGPU_BF16 && p.c.dtype != DFGPU_F16 && p.c.dtype != DFGPU_F32 && p.c.dtype != DFGPU_E4M3 && p.c.dtype != DFGPU_E5M2) return false;
    if (!describe(p.a, p.b, p.c, kCodes, problem)) return false;
    // f32 results, but for whole tiles in whole 16-byte units (which always came from one accumulator): the blocks summed in f32. Relative
    // error at 2050 x 256 / 640 x 1040: 1.36 / 2.63e-8 by the CUDA cores' additions, 1.5 / 3.22e-8 in one accumulator, 1.27 / 2.2e-8 this way.
    const bool whole = problem.M % 128 == 0 && problem.N % 128 == 0 && problem.K % 128 == 0 && problem.c_ld % 4 == 0;
    if (p.c.dtype == DFGPU_F32 && !whole) problem.kind = kCodesSummed;
    return true;
}

bool matmul_fp8_tiles_supported(const dfgpu_matmul_fp8_params& p) {
    Problem problem;
    return fp8_problem(p, problem);
}

// What the kernel id DFGPU_MATMUL_FP8_UMMA promises: whole tiles and the outputs it names.
bool matmul_fp8_umma_supported(const dfgpu_matmul_fp8_params& p) {
    Problem problem;
    return fp8_problem(p, problem) && problem.M % 128 == 0 && problem.N % 128 == 0 && problem.K % 128 == 0 && p.c.dtype != DFGPU_F16 && p.c.dtype != DFGPU_E5M2;
}

int launch_matmul_fp8_umma(const dfgpu_matmul_fp8_params& p, void* const* tensors, cudaStream_t stream) {
    Problem problem;
    TileArgs args{};
    if (!on16(tensors[0]) || !on16(tensors[1])) return fail(kInvalidArgument, "MATMUL_FP8: the tcgen05 kernel needs 16-byte aligned A and B");
    if (!fp8_problem(p, problem)) return fail(kUnsupported, "MATMUL_FP8: the tcgen05 kernel does not take these operands");
    args.idesc = (p.a.dtype == DFGPU_E5M2 ? 1u << 7 : 0u) | (p.b.dtype == DFGPU_E5M2 ? 1u << 10 : 0u);
    args.amax_bits = static_cast<unsigned int*>(tensors[3]);
    args.descale_a = static_cast<const float*>(tensors[4]);
    args.descale_b = static_cast<const float*>(tensors[5]);
    args.scale_c = static_cast<const float*>(tensors[6]);
    return launch_problem(problem, args, tensors[0], tensors[1], tensors[2], stream, "MATMUL_FP8 (tcgen05)");
}

int matmul_tiles_device_status(int* status) { return read_and_clear_device_status(status); }

}  // namespace dfgpu
