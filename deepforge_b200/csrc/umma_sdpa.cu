// SDPA forward on the 5th-generation tensor cores: bf16 or f16, head dimension 64 or 128, any sequence lengths, grouped heads,
// causal (top-left) and padding masks.
//
// The running maximum is only raised when it grows by more than 2^8 (the accumulator is rescaled
// in TMEM then, which is rare); Stats = ln2 * (m + log2(l)) is exact whichever reference m is
// in use. Causal graphs skip tiles above the diagonal and mask inside the diagonal tile.
// Scores are scaled after the f32 dot product, invalid positions are -inf, as in the reference's
// emit_sdpa_forward (lib/Compiler/SequenceGraph.cpp:2135-2341).
//
// Lengths are free because the copies are: Q, K, V and O are rank-4 tensor maps (channel, position, head, batch), so TMA fills
// the positions past the end with zeros and clips them on the store, and what is left is a mask on the last key tile. With
// SEQ_LEN_Q / SEQ_LEN_KV a batch's key tiles end at its own length, V rows behind it are cleared in shared memory (a zero
// probability times an infinity in the padding would be NaN), and rows past SEQ_LEN_Q store 0 and -inf. 4 x 16 heads of 1000
// padded positions, causal: 9.7 ms on the row-at-a-time kernel, 26 to 34 us here, by the lengths (before the halves and the order below 36;
// 31 then with P in one 16-bit piece, and O 1.33 times as far from 64 bits).
#include <algorithm>
#include <cmath>

#include "umma_ptx.cuh"

namespace dfgpu {
namespace {

constexpr int kRows = 128;      // query rows per CTA
constexpr int kKeys = 128;      // keys per tile
constexpr float kRescaleThreshold = 8.0f;  // log2 units

struct SdpaUmmaArgs {
    int32_t heads_q, heads_kv, seq_q, seq_kv;
    int32_t pairs;            // of 128-row query tiles, the last one perhaps partly past the end
    int32_t causal;
    int32_t order;            // of the work list: kAsStored, kHeavyWithLight, kHeaviestFirst or kLongestFirst (see PairWalker)
    float scale_log2;  // |attn_scale| * log2(e); a negative scale negates Q in the products
    uint32_t negate_q; // ... through this bit of the instruction descriptor
    const int32_t* len_q;   // SEQ_LEN_Q and SEQ_LEN_KV by batch, or null
    const int32_t* len_kv;
    int64_t len_q_stride, len_kv_stride;
    float* stats;      // [B, Hq, Sq] or null
    int64_t stats_batch_stride, stats_head_stride, stats_row_stride;
    // Max and Sum_exp rows, or null; element strides like Stats
    float* row_max;
    float* row_sum;
    int64_t max_stride[3], sum_stride[3];
    float attn_scale;  // |attn_scale|, natural-log units: Max = attn_scale * largest dot product
    float to_natural[2];  // attn_scale / scale_log2 as a sum: what takes m_ref to natural-log units
    int32_t batch_heads;  // batch * query heads
};

__device__ __forceinline__ void tmem_store_16(uint32_t taddr, const uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
          "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
}
__device__ __forceinline__ void tmem_store_8(uint32_t taddr, const uint32_t (&r)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                 ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
                 : "memory");
}
__device__ __forceinline__ void tmem_store_4(uint32_t taddr, const uint32_t (&r)[4]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};" ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]) : "memory");
}
__device__ __forceinline__ void tmem_store_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// ---- two query tiles per CTA ------------------------------------------------------
// The softmax of one tile costs about as many cycles as its two products, so a CTA that owns two
// 128-row query tiles (A and B) lets the tensor pipe work on one while the other is in its softmax:
//   warp 16     TMA: Q_A, Q_B once, then K_0, V_0, K_1, ... into a ring of 32 KiB slots
//   warp 17     one lane issues, per key tile j:  O_A += P_A(j) V_j ; S_A(j+1) = Q_A K_{j+1}^T ;
//                                                 O_B += P_B(j) V_j ; S_B(j+1) = Q_B K_{j+1}^T
//   warps 0-7   softmax of tile A, warps 8-15 softmax of tile B: two threads per query row, each with 64 of the
//               tile's 128 keys (the two warps that share a lane quarter trade row maxima through shared memory)
// Probabilities are handed over in two halves, each thread's first 32 keys under the exponentials of its others: a tile's chain of score
// product, softmax and second product is what a round waits for (8 x 32 x 2048 x 128 causal 334 -> 329 us, 12 heads of 2061 x 64 causal
// 40.1 -> 37.3, 2 x 32 x 4000 x 64 padded 178 -> 167).
// (D is the head dimension.) TMEM: S_A at +0, S_B at +128, O_A at +256, O_B at +384. P never goes through shared memory: each
// thread overwrites its own score row with the 16-bit probabilities (two per 32-bit
// column) and the second product takes its A operand from tensor memory. The tensor pipe runs the
// products of one CTA in issue order, so S_X(j+1) may be issued right behind the product that reads P_X(j).
// Under a causal mask tile A (the earlier rows) has one key tile fewer than tile B.

constexpr int kPairSlots = 4;
constexpr int kPolyEvery = 4;  // one pair of exponentials in kPolyEvery goes to the FMA pipe (0: none)
constexpr int kPairThreads = 608;  // 2 x 8 softmax warps (two threads per query row), loader, issuer and output-store warps

template <int D>
struct PairSmem {
    static constexpr int kTile = kRows * D * 2;         // one Q / K / V / O tile: D / 64 boxes of 128 rows x 64 channels
    static constexpr int kQ = 0;                       // Q_A, Q_B
    static constexpr int kRing = 2 * kTile;
    static constexpr int kStage = kRing + kPairSlots * kTile;  // one output tile on its way to global memory
    // 128 bytes per (tile, lane quarter): during the key loop the half-row maxima [half][lane] as bf16, after it the row sum
    // [lane] as f32; GENERAL: behind them the maxima's third bytes (f32 maxima would not fit beside two Q tiles, four 32 KiB ring
    // slots and the output tile).
    static constexpr int kExchange = kStage + kTile;
    static constexpr int kBarriers = kExchange + 1024 + 512;
    // stage_free, q_full[2], q_empty[2], kv_full[S], kv_empty[S], s_full[2], p_full[2], o_full[2], o_empty[2], staged[2], p_half[2]
    static constexpr int kBarrierCount = 5 + 2 * kPairSlots + 12;
    static constexpr int kList = kBarriers + kBarrierCount * 8 + 16;   // kLongestFirst: kMostPairs bytes
    static constexpr int kMostPairs = 256;
    static constexpr int kTotal = kList + kMostPairs;
    static constexpr int kDynamic = kTotal + 1024;
    static_assert(kDynamic <= 227 * 1024, "the most a block may have");
};
constexpr int kHalfBytes = kRows * 128;   // one box


// D[tmem] (+)= A[tmem] * B[smem]: the A operand (bf16 pairs, one row per lane) is read from tensor memory.
__device__ __forceinline__ void umma_bf16_a_tmem(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate) : "memory");
}

__device__ __forceinline__ float ex2_fast(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// Packed pairs of f32 (one 64-bit register): Blackwell's FMA pipe takes two lanes per instruction, which
// halves the instruction count of the scale-and-subtract and of the row sums in the softmax loop.
__device__ __forceinline__ uint64_t pack2(float lo, float hi) {
    uint64_t v;
    asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(lo), "f"(hi));
    return v;
}
__device__ __forceinline__ void unpack2(uint64_t v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
    uint64_t d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}

// 2^x on the FMA and integer pipes: round x to the nearest integer n with the 1.5 * 2^23 trick, evaluate a
// cubic for 2^(x - n) on [-0.5, 0.5] (relative error 7.5e-5, far below the bf16 rounding of P) and add n
// to the exponent field. The special-function unit runs 16 ex2 per clock per SM: 1024 cycles for a 128 x 128
// score tile, as long as its two tensor-core products take, so part of the exponentials go this way.
// On a packed pair: the range reduction and the cubic run as f32x2 instructions (6 per pair), only the clamp and the
// exponent insertion are per element. Masked scores (-inf) end as 2^-125: nothing in a sum that holds a term >= 2^-8.
__device__ __forceinline__ void exp2_poly_pair(uint64_t x2, float& p0, float& p1) {
    float x0, x1;
    unpack2(x2, x0, x1);
    x2 = pack2(fmaxf(x0, -125.0f), fmaxf(x1, -125.0f));
    const uint64_t magic2 = pack2(12582912.0f, 12582912.0f);
    const uint64_t t2 = add2(x2, magic2);
    const uint64_t n2 = add2(t2, pack2(-12582912.0f, -12582912.0f));
    const uint64_t f2 = fma2(n2, pack2(-1.0f, -1.0f), x2);
    uint64_t q2 = fma2(pack2(0.0551716685f, 0.0551716685f), f2, pack2(0.2426111251f, 0.2426111251f));
    q2 = fma2(q2, f2, pack2(0.6932609677f, 0.6932609677f));
    q2 = fma2(q2, f2, pack2(0.9999280572f, 0.9999280572f));
    float q0, q1, t0, t1;
    unpack2(q2, q0, q1);
    unpack2(t2, t0, t1);
    p0 = __int_as_float(__float_as_int(q0) + (__float_as_int(t0) << 23));
    p1 = __int_as_float(__float_as_int(q1) + (__float_as_int(t1) << 23));
}

__device__ __forceinline__ void tmem_load_16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr) : "memory");
}
// Wait for the tensor-memory loads in flight. The registers of the load that is about to be used pass through the
// statement, so that nothing that reads them can be scheduled above the wait while a later load is already in flight.
__device__ __forceinline__ void tmem_load_wait_for(uint32_t (&r)[16]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
                   "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15])
                 :: "memory");
}
__device__ __forceinline__ float max3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
// Largest of 16 scores folded into `running`: eight three-input maxima.
__device__ __forceinline__ float max_of_16(const uint32_t (&raw)[16], float running) {
    float part[4];
#pragma unroll
    for (int g = 0; g < 4; ++g)
        part[g] = max3(__uint_as_float(raw[4 * g]), __uint_as_float(raw[4 * g + 1]), max3(__uint_as_float(raw[4 * g + 2]), __uint_as_float(raw[4 * g + 3]), running));
    return fmaxf(fmaxf(part[0], part[1]), fmaxf(part[2], part[3]));
}
template <bool F16>
__device__ __forceinline__ uint32_t pack_pair(float lo, float hi) {
    if constexpr (F16) {
        const __half2 two = __floats2half2_rn(lo, hi);
        return *reinterpret_cast<const uint32_t*>(&two);
    } else {
        const __nv_bfloat162 two = __floats2bfloat162_rn(lo, hi);
        return *reinterpret_cast<const uint32_t*>(&two);
    }
}
template <bool F16>
__device__ __forceinline__ void unpack_pair(uint32_t two, float& lo, float& hi) {
    if constexpr (F16) {
        const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&two));
        lo = f.x;
        hi = f.y;
    } else {
        lo = __uint_as_float(two << 16);
        hi = __uint_as_float(two & 0xffff0000u);
    }
}
// Sixteen scores -> probabilities 2^(s * scale + bias) as bf16 or f16 pairs in tensor memory, their sum added to two packed partial
// sums. GENERAL: every exponential by the special-function unit (2^-22), and eight columns behind each pair what its rounding left
// over, eight scores at a time (sixteen at once spilled).
template <bool F16, bool GENERAL>
__device__ __forceinline__ void put_probabilities(const uint32_t (&raw)[16], uint64_t scale2, uint64_t bias2, uint64_t (&sums)[2], uint32_t address) {
    constexpr int kParts = GENERAL ? 2 : 1, kPairs = 8 / kParts;
#pragma unroll
    for (int part = 0; part < kParts; ++part) {
        uint32_t packed[kPairs], left[kPairs];
#pragma unroll
        for (int e = 0; e < kPairs; ++e) {
            const int i = part * kPairs + e;
            const uint64_t v = fma2(pack2(__uint_as_float(raw[2 * i]), __uint_as_float(raw[2 * i + 1])), scale2, bias2);
            float p0, p1;
            if (!GENERAL && kPolyEvery > 0 && i % (kPolyEvery > 0 ? kPolyEvery : 1) == 0) {
                exp2_poly_pair(v, p0, p1);  // this pair on the FMA pipe
            } else {
                float x0, x1;
                unpack2(v, x0, x1);
                p0 = ex2_fast(x0);
                p1 = ex2_fast(x1);
            }
            sums[i & 1] = add2(sums[i & 1], pack2(p0, p1));
            packed[e] = pack_pair<F16>(p0, p1);
            if constexpr (GENERAL) {
                float head0, head1;
                unpack_pair<F16>(packed[e], head0, head1);
                left[e] = pack_pair<F16>(p0 - head0, p1 - head1);
            }
        }
        if constexpr (GENERAL) {
            tmem_store_4(address + part * 4, packed);
            tmem_store_4(address + 8 + part * 4, left);
        } else {
            tmem_store_8(address, packed);
        }
    }
}
// The upper BITS bits of a float, rounded towards +inf.
template <int BITS>
__device__ __forceinline__ uint32_t round_up(float value) {
    constexpr uint32_t kDropped = (1u << (32 - BITS)) - 1u;
    const uint32_t bits = __float_as_uint(value);
    return (bits & 0x80000000u) ? bits & ~kDropped : (bits + kDropped) & ~kDropped;
}
// What is added to the scaled scores of a row. (GENERAL: scores that are all -inf are probabilities of zero, not NaN.)
template <bool GENERAL>
__device__ __forceinline__ float bias_of(float m_ref) { return GENERAL && m_ref == -INFINITY ? 0.0f : -m_ref; }
template <bool GENERAL>
__device__ __forceinline__ float inverse_of(float total) { return GENERAL && !(total > 0.0f) ? 0.0f : 1.0f / total; }
// Sum_exp: the sum was accumulated against m_ref; re-express it against the true maximum.
template <bool GENERAL>
__device__ __forceinline__ float sum_against(float total, float m_ref, float row_max) { return GENERAL && total == 0.0f ? 0.0f : total * exp2f(m_ref - row_max); }
// Stats of a row whose probabilities were formed against m_ref.
template <bool GENERAL>
__device__ __forceinline__ float natural_log_sum(const SdpaUmmaArgs& args, float m_ref, float total) {
    // (rounded once behind the logarithm, as the row-at-a-time kernel's)
    if constexpr (GENERAL) return m_ref == -INFINITY ? m_ref : fmaf(m_ref, args.to_natural[0], fmaf(m_ref, args.to_natural[1], logf(total)));
    return 0.6931471805599453f * (m_ref + log2f(total));
}
// Columns that put_probabilities() fills for 16 keys.
template <bool GENERAL>
constexpr int kProbabilityColumns = GENERAL ? 16 : 8;

// One (batch, head, query pair) of the work list.
struct PairItem {
    int batch, head, kv_head;
    int q_tile_a;        // index of the first of the two 128-row query tiles
    int tiles_a, tiles_b;  // key tiles the two query tiles walk (up to their diagonals and the batch's length), at least one
    int tiles;           // ... the larger of them: key tiles that are loaded
    int kv_len;          // keys of this batch, at least one
    int live_q;          // query rows before this one have keys; the others store 0 and -inf
};

// GENERAL: what the kernels take beyond whole tiles of packed bf16 rows of 128 (plain_tiles()): a batch's keys may end inside a key
// tile (padding masks, or a key length that is no multiple of 128), and probabilities are held to f32's accuracy: O += P V runs
// twice, on P rounded to the operands' type and on what that left over (16 or 22 bits in all), as O and Stats of these graphs are
// those of f32 probabilities (sdpa_rowwise_kernel's) to the rounding of O. Without it the masks of the last tile, the clearing of V
// rows and the dead rows are not compiled in: they cost 5 % of 8 x 32 x 2048 causal. (LENGTHS: the batches have lengths of their own.)
template <bool LENGTHS>
__device__ __forceinline__ PairItem pair_item(const SdpaUmmaArgs& args, int bh, int pair) {
    PairItem item;
    item.batch = bh / args.heads_q;
    item.head = bh - item.batch * args.heads_q;
    item.kv_head = item.head / (args.heads_q / args.heads_kv);
    item.q_tile_a = 2 * pair;
    item.kv_len = args.seq_kv;
    item.live_q = args.seq_q;
    if (LENGTHS && args.len_q != nullptr) {
        const int len_kv = args.len_kv[item.batch * args.len_kv_stride];
        item.live_q = len_kv > 0 ? min(item.live_q, args.len_q[item.batch * args.len_q_stride]) : 0;
        item.kv_len = max(1, min(item.kv_len, len_kv));
    }
    const int kv_tiles = (item.kv_len + kKeys - 1) / kKeys;
    auto tiles_of = [&](int q_tile) {
        if (q_tile * kRows >= item.live_q) return 1;
        return args.causal ? min(kv_tiles, q_tile + 1) : kv_tiles;
    };
    item.tiles_a = tiles_of(item.q_tile_a);
    item.tiles_b = tiles_of(item.q_tile_a + 1);
    item.tiles = max(item.tiles_a, item.tiles_b);
    return item;
}

// The work list of one CTA (or cluster), the same in every warp role.
//   kAsStored        every query pair of a head is a unit
//   kHeavyWithLight  causal, one SM per pair: unit i of a head is the heavy pair P-1-i followed by the light pair i, so that every unit
//                    walks 2P+2 key tiles and equal numbers of units are equal work
//   kHeaviestFirst   causal, two SMs per pair: the pairs of all heads by falling length, and every other round
//                    in reverse, so that the CTA with the longest pair of one round gets the shortest of the next
//   kLongestFirst    padded lengths, one SM per pair: the same by the key tiles that a batch's own lengths leave of its pairs, in an order
//                    that each CTA works out for itself (longest_first()). 4 x 16 heads of 500 to 1000 positions causal: 8 key tiles on the
//                    longest list instead of 10, 34.7 -> 26.2 us with the halves above; 2 x 32 x 4000 x 64 252 -> 178 by the order alone.
// CTA c takes units c, c + gridDim.x, ...; but for the last order neighbouring CTAs thus work on the same head at the same
// time and share its K and V in L2.
enum { kAsStored = 0, kHeavyWithLight = 1, kHeaviestFirst = 2, kLongestFirst = 3 };
template <int CTAS, bool LISTED = false>   // CTAs that walk one list together; LISTED: kLongestFirst is compiled in (it cost the other orders 2 %)
struct PairWalker {
    int k = 0;
    const uint8_t* list = nullptr;   // kLongestFirst: (batch, pair) by falling length
    __device__ __forceinline__ bool next(const SdpaUmmaArgs& args, int& bh, int& pair) {
        const int pairs = args.pairs;
        if constexpr (CTAS == 2) {
            const int places = static_cast<int>(gridDim.x) / CTAS, place = static_cast<int>(blockIdx.x) / CTAS;   // (the grid is a multiple of CTAS)
            const bool heaviest_first = args.order == kHeaviestFirst;
            const int unit = k * places + (heaviest_first && (k & 1) ? places - 1 - place : place);
            ++k;
            if (unit >= pairs * args.batch_heads) return false;   // (a reversed last round may have nothing for this place)
            if (heaviest_first) {
                pair = unit / args.batch_heads;
                bh = unit - pair * args.batch_heads;
                pair = pairs - 1 - pair;
            } else {
                bh = unit / pairs;
                pair = unit - bh * pairs;
            }
            return true;
        }
        if (LISTED && args.order == kLongestFirst) {
            const int places = static_cast<int>(gridDim.x), place = static_cast<int>(blockIdx.x);
            const int unit = k * places + ((k & 1) ? places - 1 - place : place);
            ++k;
            if (unit >= pairs * args.batch_heads) return false;
            const int at = unit / args.heads_q, entry = list[at], batch = entry / pairs;
            bh = batch * args.heads_q + unit - at * args.heads_q;
            pair = entry - batch * pairs;
            return true;
        }
        const int units_per_head = args.order == kHeavyWithLight ? (pairs + 1) >> 1 : pairs;
        const int units = units_per_head * args.batch_heads;
        for (;; ++k) {
            const int unit = static_cast<int>(blockIdx.x) + (k >> 1) * static_cast<int>(gridDim.x);
            if (unit >= units) return false;
            bh = unit / units_per_head;
            const int i = unit - bh * units_per_head;
            pair = i;
            if (args.order == kHeavyWithLight) {
                pair = (k & 1) ? i : pairs - 1 - i;
                if ((k & 1) && 2 * i == pairs - 1) continue;  // the middle pair of an odd count stands alone
            } else if (k & 1) {
                continue;
            }
            ++k;
            return true;
        }
    }
};
// The (batch, pair)s, at most 256, by falling number of key tiles: every thread counts the ones ahead of its own.
__device__ __forceinline__ void longest_first(const SdpaUmmaArgs& args, uint8_t* list, uint16_t* weights) {
    const int count = args.batch_heads / args.heads_q * args.pairs, own = static_cast<int>(threadIdx.x);
    int weight = 0;
    if (own < count) {
        const int batch = own / args.pairs;
        const PairItem item = pair_item<true>(args, batch * args.heads_q, own - batch * args.pairs);
        weight = item.tiles_a + item.tiles_b;
        weights[own] = static_cast<uint16_t>(weight);
    }
    __syncthreads();
    if (own < count) {
        int ahead = 0;
        for (int i = 0; i < count; ++i) ahead += weights[i] > weight || (weights[i] == weight && i < own) ? 1 : 0;
        list[ahead] = static_cast<uint8_t>(own);
    }
    __syncthreads();
}
template <int CTAS, bool LISTED, class Body>
__device__ __forceinline__ void for_each_pair_item(const SdpaUmmaArgs& args, const uint8_t* list, Body&& body) {
    PairWalker<CTAS, LISTED> walker;
    walker.list = list;
    int bh, pair;
    while (walker.next(args, bh, pair))  // one call site of the body: it is a whole warp role
        if (!body(bh, pair)) return;
}

// Persistent form: one CTA per SM walks its work list, and the prologue of an item (Q and the first K/V tiles, the
// first score products) runs under the tail of the previous one. 19 warps:
//   warps 0-15  softmax, two threads per query row (8 warps per query tile); they also normalise O into a staging tile
//   warp 16     TMA producer: Q_A and Q_B of an item as soon as the previous item's last score product has read the
//               old ones, then K_0, V_0, K_1, ... through a ring of 32 KiB slots that runs on across items
//   warp 17     issues the products; one elected lane issues, all lanes walk the schedule
//   warp 18     sends staged output tiles to global memory by TMA (row-per-thread global stores of 16 bytes at a
//               256-byte stride kept the load/store unit busy for ~5000 cycles per tile)
template <int D, bool F16, bool GENERAL, bool PADDED>
__global__ void __launch_bounds__(kPairThreads, 1)
sdpa_umma_pair_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                      const __grid_constant__ CUtensorMap map_v, const __grid_constant__ CUtensorMap map_o, SdpaUmmaArgs args) {
    using Smem = PairSmem<D>;
    constexpr int kTileBytes = Smem::kTile;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t* generic_base = smem_raw + (smem_base - smem_u32(smem_raw));
    const uint32_t bar_base = smem_base + Smem::kBarriers;
    const uint32_t stage_free = bar_base;
    auto q_full = [&](int x) { return bar_base + 8u * (1 + x); };
    auto q_empty = [&](int x) { return bar_base + 8u * (3 + x); };
    auto kv_full = [&](int s) { return bar_base + 8u * (5 + s); };
    auto kv_empty = [&](int s) { return bar_base + 8u * (5 + kPairSlots + s); };
    auto s_full = [&](int x) { return bar_base + 8u * (5 + 2 * kPairSlots + x); };
    auto p_full = [&](int x) { return bar_base + 8u * (7 + 2 * kPairSlots + x); };
    auto o_full = [&](int x) { return bar_base + 8u * (9 + 2 * kPairSlots + x); };
    auto o_empty = [&](int x) { return bar_base + 8u * (11 + 2 * kPairSlots + x); };
    auto staged = [&](int x) { return bar_base + 8u * (13 + 2 * kPairSlots + x); };
    auto p_half = [&](int x) { return bar_base + 8u * (15 + 2 * kPairSlots + x); };
    const uint32_t tmem_slot = bar_base + 8u * Smem::kBarrierCount;
    volatile uint32_t* tmem_slot_ptr = reinterpret_cast<volatile uint32_t*>(generic_base + Smem::kBarriers + 8 * Smem::kBarrierCount);

    const int warp = uniform_warp_index(), lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        prefetch_tensormap(&map_q);
        prefetch_tensormap(&map_k);
        prefetch_tensormap(&map_v);
        prefetch_tensormap(&map_o);
        mbar_init(stage_free, 1);
        for (int s = 0; s < kPairSlots; ++s) {
            mbar_init(kv_full(s), 1);
            mbar_init(kv_empty(s), 1);
        }
        for (int x = 0; x < 2; ++x) {
            mbar_init(s_full(x), 1);
            mbar_init(p_half(x), 8);
            mbar_init(p_full(x), 8);
            mbar_init(o_full(x), 1);
            mbar_init(q_full(x), 1);
            mbar_init(q_empty(x), 1);
            mbar_init(o_empty(x), 8);
            mbar_init(staged(x), 8);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 17) {
        tmem_alloc(tmem_slot, 512);
        tmem_relinquish();
        tc_fence_before();
    }
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot_ptr;
    chain_wait();
    const uint8_t* list = PADDED ? generic_base + Smem::kList : nullptr;
    if (PADDED && args.order == kLongestFirst) longest_first(args, generic_base + Smem::kList, reinterpret_cast<uint16_t*>(generic_base + Smem::kStage));
    // (no early release: this kernel fills every SM, so the next one's CTAs would only wait beside it, 0.6 % of 330 us)

    if (warp == 16) {
        const bool leader = elect_one();
        int slot = 0;
        uint32_t phase = 1;  // parity of the "slot is free" wait
        uint32_t n = 0;      // items started
        for_each_pair_item<1, PADDED>(args, list, [&](int bh, int pair) {
            const PairItem item = pair_item<PADDED>(args, bh, pair);
            auto load_box = [&](uint32_t dst, const CUtensorMap* map, int row, int head, uint32_t bar) {
#pragma unroll
                for (int h = 0; h < D / 64; ++h) tma_load_4d(dst + h * kHalfBytes, map, 64 * h, row, head, item.batch, bar);
            };
            // a Q buffer is free once the previous item's last score product of that query tile has completed; tile A's
            // (which under a causal mask ends a key tile earlier) and the first K tile go first, so that the issuing warp
            // can start this item's tile A under the previous item's last round
            auto load_q = [&](int x) {
                if (!mbar_wait_warp(q_empty(x), (n & 1) ^ 1, 220 + x)) return false;
                if (leader) {
                    mbar_expect_tx(q_full(x), kTileBytes);
                    load_box(smem_base + Smem::kQ + x * kTileBytes, &map_q, (item.q_tile_a + x) * kRows, item.head, q_full(x));
                }
                return true;
            };
            if (!load_q(0)) return false;
            for (int t = 0; t < 2 * item.tiles; ++t) {
                if (t == 1 && !load_q(1)) return false;
                if (!mbar_wait_warp(kv_empty(slot), phase, 215)) return false;
                const uint32_t dst = smem_base + Smem::kRing + slot * kTileBytes;
                if (leader) {
                    mbar_expect_tx(kv_full(slot), kTileBytes);
                    load_box(dst, (t & 1) ? &map_v : &map_k, (t >> 1) * kKeys, item.kv_head, kv_full(slot));
                }
                if (++slot == kPairSlots) { slot = 0; phase ^= 1; }
            }
            ++n;
            return true;
        });
    } else if (warp == 17) {
        // All 32 lanes walk the schedule; the elected lane issues the products and their commits.
        const bool leader = elect_one();
        // f32 accumulators, bf16 (1) or f16 (0) operands, N, M; the second product reads V MN-major
        constexpr uint32_t kFormats = (1u << 4) | (F16 ? 0u : (1u << 7) | (1u << 10)) | (static_cast<uint32_t>(kRows >> 4) << 24);
        const uint32_t idesc_qk = kFormats | (static_cast<uint32_t>(kKeys >> 3) << 17) | args.negate_q;
        constexpr uint32_t idesc_pv = kFormats | (static_cast<uint32_t>(D >> 3) << 17) | (1u << 16);
        const uint32_t tmem_u = __shfl_sync(0xffffffffu, tmem_base, 0);
        bool ok = true;
        int slot = 0;         // ring slot of the next K or V tile to consume
        uint32_t phase = 0;
        uint32_t n = 0;       // items started
        uint32_t p_count[2] = {0, 0};  // probability tiles consumed per query tile (parity of p_full)
        // (no tcgen05 fence after a slot wait: the slot was filled by TMA, not by tensor-memory traffic of other threads)
        auto wait_slot = [&](int code) {
            if (ok) ok = mbar_wait_warp(kv_full(slot), phase, code);
        };
        auto next_slot = [&]() { if (++slot == kPairSlots) { slot = 0; phase ^= 1; } };
        auto commit = [&](uint32_t bar) { if (leader) umma_commit(bar); };
        constexpr uint32_t kDescHi = smem_desc_hi(1024);
        auto scores = [&](int x, int k_slot) {  // S_x = Q_x K^T
            if (!ok) return;
            const uint32_t q_lo = smem_desc_lo(smem_base + Smem::kQ + x * kTileBytes, 16);
            const uint32_t k_lo = smem_desc_lo(smem_base + Smem::kRing + k_slot * kTileBytes, 16);
            const uint32_t d_tmem = tmem_u + x * 128;
            if (leader) {
#pragma unroll
                for (int k = 0; k < D / 16; ++k) {
                    const uint32_t offset = ((k >> 2) * kHalfBytes + (k & 3) * 32) >> 4;  // in 16-byte units
                    umma_bf16(d_tmem, desc_words(q_lo + offset, kDescHi), desc_words(k_lo + offset, kDescHi), idesc_qk, k != 0 ? 1u : 0u);
                }
            }
        };
        // O_x += P_x V_j. P_x lies as 16-bit pairs over the scores: keys 0..63 in columns 0..31 of S_x, keys 64..127 in columns
        // 64..95 (each softmax thread overwrites columns that held its own scores only); GENERAL: every 16 keys' pairs and then
        // their left-overs over those keys' 16 scores, so columns 0..63 and 64..127. The first product of an item
        // overwrites O_x, which the softmax warps must have read out for the previous item.
        auto product = [&](int x, int j, int v_slot) {
            if (ok && j == 0) ok = mbar_wait_warp(o_empty(x), (n & 1) ^ 1, 218 + x);
            // (in two halves: the first 32 of each thread's 64 keys are multiplied while the softmax warps form the others)
            const uint32_t v_lo = smem_desc_lo(smem_base + Smem::kRing + v_slot * kTileBytes, kHalfBytes);
            const uint32_t d_tmem = tmem_u + 256 + x * 128, p_tmem = tmem_u + x * 128;
#pragma unroll
            for (int part = 0; part < 2; ++part) {
                if (ok) ok = mbar_wait_warp(part == 0 ? p_half(x) : p_full(x), p_count[x] & 1, 223 + x);
                tc_fence_after();
                if (leader && ok) {
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const int k = (i >> 1) * 4 + part * 2 + (i & 1);   // 16 keys
                        const uint32_t p_at = p_tmem + (k >> 2) * 64 + (k & 3) * kProbabilityColumns<GENERAL>;
                        umma_bf16_a_tmem(d_tmem, p_at, desc_words(v_lo + ((k * 2048) >> 4), kDescHi), idesc_pv, (j | k) != 0 ? 1u : 0u);
                        if constexpr (GENERAL) umma_bf16_a_tmem(d_tmem, p_at + 8, desc_words(v_lo + ((k * 2048) >> 4), kDescHi), idesc_pv, 1u);
                    }
                }
            }
            ++p_count[x];
        };
        PairWalker<1, PADDED> walker;
        walker.list = list;
        int bh = 0, pair = 0, next_bh = 0, next_pair = 0;
        bool have = walker.next(args, bh, pair);
        bool early = false;  // S_A of the current item was issued in the previous item's last round
        int early_slot = 0;  // the ring slot of its K tile
        while (have && ok) {
            const PairItem item = pair_item<PADDED>(args, bh, pair);
            const int tiles_a = item.tiles_a, tiles_b = item.tiles_b, tiles = item.tiles;
            const bool have_next = walker.next(args, next_bh, next_pair);
            const int next_tiles_a = have_next ? pair_item<PADDED>(args, next_bh, next_pair).tiles_a : 0;
            int k0_slot = early_slot;
            if (!early) {
                if (ok) ok = mbar_wait_warp(q_full(0), n & 1, 222);
                wait_slot(225);
                k0_slot = slot;
                next_slot();
                scores(0, k0_slot);
                commit(s_full(0));
                if (tiles_a == 1) commit(q_empty(0));
            }
            early = false;
            if (ok) ok = mbar_wait_warp(q_full(1), n & 1, 214);
            scores(1, k0_slot);
            commit(s_full(1));
            commit(kv_empty(k0_slot));
            if (tiles_b == 1) commit(q_empty(1));
            for (int j = 0; j < tiles; ++j) {
                wait_slot(226);
                const int v_slot = slot;
                next_slot();
                if (j < tiles_a) {
                    product(0, j, v_slot);
                    if (j == tiles_a - 1) commit(o_full(0));
                } else if (have_next && ok && j == tiles - 1) {
                    // Tile A has no key tile in this item's last round (causal mask): if the next item's Q_A and first K
                    // tile have landed, its first scores go out now and its softmax runs under tile B's last round.
                    const bool landed = __all_sync(0xffffffffu, mbar_test_wait(q_full(0), (n + 1) & 1)) && __all_sync(0xffffffffu, mbar_test_wait(kv_full(slot), phase));
                    if (landed) {
                        early = true;
                        early_slot = slot;
                        next_slot();
                        scores(0, early_slot);
                        commit(s_full(0));
                        if (next_tiles_a == 1) commit(q_empty(0));
                    }
                }
                const bool more = j + 1 < tiles;
                int k_slot = 0;
                if (more) {
                    wait_slot(227);
                    k_slot = slot;
                    next_slot();
                }
                if (j + 1 < tiles_a) {
                    scores(0, k_slot);
                    commit(s_full(0));
                    if (j + 2 == tiles_a) commit(q_empty(0));  // the item's last read of Q_A
                }
                if (j < tiles_b) {
                    product(1, j, v_slot);
                    if (j == tiles_b - 1) commit(o_full(1));
                }
                commit(kv_empty(v_slot));
                if (j + 1 < tiles_b) {
                    scores(1, k_slot);
                    commit(s_full(1));
                    if (j + 2 == tiles_b) commit(q_empty(1));  // the item's last read of Q_B
                }
                if (more) commit(kv_empty(k_slot));
            }
            ++n;
            bh = next_bh;
            pair = next_pair;
            have = have_next;
        }
    } else if (warp == 18) {
        // Output stores: a query tile's softmax warps leave the normalised tile in the staging buffer; this warp sends it
        // off and hands the buffer to the next tile once the copy engine has read it.
        const bool leader = elect_one();
        uint32_t n = 0;
        bool ok = true;
        for_each_pair_item<1, PADDED>(args, list, [&](int bh, int pair) {
            const PairItem item = pair_item<PADDED>(args, bh, pair);
            for (int x = 0; x < 2; ++x) {
                if (ok) ok = mbar_wait_warp(staged(x), n & 1, 216 + x);
                if (leader) {
                    if (ok && g_device_status == 0) {
                        const int row = (item.q_tile_a + x) * kRows;
                        if (row < args.seq_q) {
#pragma unroll
                            for (int h = 0; h < D / 64; ++h) tma_store_4d(&map_o, smem_base + Smem::kStage + h * kHalfBytes, 64 * h, row, item.head, item.batch);
                        }
                    }
                    tma_store_commit();
                    tma_store_wait_read<0>();
                    mbar_arrive(stage_free);
                }
                __syncwarp();
            }
            ++n;
            return true;
        });
        if (leader) tma_store_wait_all();
    } else {
        const int sw = warp;
        const int x = sw >> 3;           // 0: tile A, 1: tile B
        const int half = (sw >> 2) & 1;  // which 64 of the tile's 128 keys (and of the 128 output columns) this thread owns
        const int quadrant = warp & 3;   // tensor-memory lane quarter of this warp; warps w and w + 4 share it
        const int row = quadrant * 32 + lane;
        const uint32_t lane_base = static_cast<uint32_t>(quadrant * 32) << 16;
        const uint32_t tmem_s = tmem_base + lane_base + x * 128;
        constexpr int kColumns = D / 2;  // of O per thread
        const uint32_t tmem_o = tmem_base + lane_base + 256 + x * 128 + half * kColumns;
        const float scale = args.scale_log2;
        const int pair_barrier = 1 + x * 4 + quadrant;  // the 64 threads that share these 32 rows
        uint16_t* exchange = reinterpret_cast<uint16_t*>(generic_base + Smem::kExchange) + ((x * 4 + quadrant) * 2) * 32;  // [half][lane]
        uint8_t* exchange_low = generic_base + Smem::kExchange + 1024 + (x * 4 + quadrant) * 64;   // [half][lane]
        float* sum_exchange = reinterpret_cast<float*>(generic_base + Smem::kExchange) + (x * 4 + quadrant) * 32;
        uint32_t n = 0;        // items started
        uint32_t s_count = 0;  // score tiles consumed (parity of s_full)
        uint32_t ring_base = 0;  // ring slots of the items before this one
        bool ok = true;
        for_each_pair_item<1, PADDED>(args, list, [&](int bh, int pair) {
        const PairItem item = pair_item<PADDED>(args, bh, pair);
        const int q_tile = item.q_tile_a + x;
        const int q_index = q_tile * kRows + row;
        const int my_tiles = x ? item.tiles_b : item.tiles_a;
        float m_ref = -INFINITY;  // reference maximum, scaled, log2 domain (identical in both threads of a row)
        float l_sum = 0.0f;       // this thread's half of the row sum
        float raw_max = -INFINITY;  // exact largest dot product among this thread's keys (for the Max / Sum_exp outputs)
        for (int j = 0; j < my_tiles; ++j, ++s_count) {
            if (ok) ok = mbar_wait(s_full(x), s_count & 1, 228 + x);
            tc_fence_after();
            // This thread's 64 scores are read twice: for the maximum, and against the reference that follows from it. (Formed in one
            // pass against the last tile's reference, probabilities wait for the exchange in registers: 2650 clocks from scores to
            // probabilities, 2270 this way.)
            // keys 0..limit of this thread's 64 are visible; only a tile at the diagonal or at the batch's end has others
            const int last_key = !GENERAL ? q_index : (args.causal ? min(q_index, item.kv_len - 1) : item.kv_len - 1);
            const int limit = last_key - j * kKeys - half * 64;
            const bool diagonal = (args.causal && j == q_tile) || (GENERAL && (j + 1) * kKeys > item.kv_len);
            const uint32_t scores_at = tmem_s + half * 64;
            auto masked = [&](uint32_t (&raw)[16], int c) {
                if (diagonal) {
#pragma unroll
                    for (int e = 0; e < 16; ++e)
                        if (c * 16 + e > limit) raw[e] = 0xff800000u;  // -inf
                }
            };
            float mine = -INFINITY;
            {
                uint32_t raw[4][16];
                tmem_load_16(scores_at, raw[0]);
                tmem_load_16(scores_at + 16, raw[1]);
#pragma unroll
                for (int c = 0; c < 4; c += 2) {
                    tmem_load_wait_for(raw[c]);
                    tmem_load_wait_for(raw[c + 1]);
                    if (c < 2) {
                        tmem_load_16(scores_at + 32, raw[2]);
                        tmem_load_16(scores_at + 48, raw[3]);
                    }
                    masked(raw[c], c);
                    masked(raw[c + 1], c + 1);
                    mine = max_of_16(raw[c + 1], max_of_16(raw[c], mine));
                }
            }
            raw_max = fmaxf(raw_max, mine);
            // Trade the half-row maxima with the warp that owns the other 64 keys of these rows, as bf16 rounded towards
            // +inf: any reference not below the true maximum by more than the threshold serves, and both threads must
            // arrive at the same value, so each uses the rounded form of its own half too. (One buffer suffices: the next
            // scores of this tile, which precede the next write, need the probabilities of all eight warps, and a warp
            // hands those over after this read.)
            // (GENERAL: as 24 bits, since against a reference 2^-7 above a maximum of thousands all probabilities would be zero)
            const uint32_t mine_up = round_up<GENERAL ? 24 : 16>(mine);
            exchange[half * 32 + lane] = static_cast<uint16_t>(mine_up >> 16);
            if (GENERAL) exchange_low[half * 32 + lane] = static_cast<uint8_t>(mine_up >> 8);
            asm volatile("bar.sync %0, 64;" ::"r"(pair_barrier) : "memory");
            uint32_t other_bits = static_cast<uint32_t>(exchange[(half ^ 1) * 32 + lane]) << 16;
            if (GENERAL) other_bits |= static_cast<uint32_t>(exchange_low[(half ^ 1) * 32 + lane]) << 8;
            const float tile_max = fmaxf(__uint_as_float(mine_up), __uint_as_float(other_bits)) * scale;
            // raise the reference only when it would grow by more than the threshold (or on the first tile); the two
            // warps of these rows see the same maxima, so they take the same branches
            if (__any_sync(0xffffffffu, tile_max > m_ref + kRescaleThreshold)) {
                const float m_new = fmaxf(m_ref, tile_max);
                const float alpha = m_ref == -INFINITY ? 0.0f : ex2_fast(m_ref - m_new);
                l_sum *= alpha;
                m_ref = m_new;
                if (j > 0) {
                    // O_x holds P V up to tile j-1; that product was issued ahead of S_x(j), which has completed.
                    // This thread rescales its columns of the row.
#pragma unroll 1
                    for (int c = 0; c < kColumns / 16; ++c) {
                        uint32_t acc[16];
                        tmem_load_16(tmem_o + c * 16, acc);
                        tmem_load_wait_for(acc);
#pragma unroll
                        for (int e = 0; e < 16; ++e) acc[e] = __float_as_uint(__uint_as_float(acc[e]) * alpha);
                        tmem_store_16(tmem_o + c * 16, acc);
                    }
                }
            }
            {
                // (probabilities go over columns whose scores have been read: 8 columns for every 16, or all 16)
                const uint64_t scale2 = pack2(scale, scale), bias2 = pack2(bias_of<GENERAL>(m_ref), bias_of<GENERAL>(m_ref));
                uint64_t sums[2] = {0, 0};  // two independent chains of packed partial sums
                uint32_t raw[4][16];
                tmem_load_16(scores_at, raw[0]);
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    tmem_load_wait_for(raw[c]);
                    if (c < 3) tmem_load_16(scores_at + (c + 1) * 16, raw[c + 1]);
                    masked(raw[c], c);
                    put_probabilities<F16, GENERAL>(raw[c], scale2, bias2, sums, scores_at + c * kProbabilityColumns<GENERAL>);
                    if (c == 1) {
                        if (PADDED && (j + 1) * kKeys > item.kv_len && (D == 128 || half == 0)) {
                            // V rows past the batch's length are not this sequence's: cleared before the product (by either tile's
                            // warps, which write the same zeros). The slot is V_j's place in the ring.
                            const uint32_t place = ring_base + 2 * j + 1, v_slot = place % kPairSlots;
                            if (ok) ok = mbar_wait(kv_full(v_slot), (place / kPairSlots) & 1, 234 + x);
                            if (j * kKeys + row >= item.kv_len) {
                                uint8_t* v_row = generic_base + Smem::kRing + v_slot * kTileBytes + half * kHalfBytes + row * 128;
#pragma unroll
                                for (int u = 0; u < 8; ++u) *reinterpret_cast<uint4*>(v_row + u * 16) = make_uint4(0, 0, 0, 0);
                            }
                            fence_async_shared();
                        }
                        tmem_store_wait();
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(p_half(x));
                    }
                }
                float lo, hi;
                unpack2(add2(sums[0], sums[1]), lo, hi);
                l_sum += lo + hi;
            }
            tmem_store_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(p_full(x));
        }
        // last product done -> read O out of tensor memory (which frees it for the next item), normalise, store
        if (ok) ok = mbar_wait(o_full(x), n & 1, 230 + x);
        tc_fence_after();
        // row sum = this thread's half + the other thread's: two hand-overs through one f32 word per row
        if (half == 1) sum_exchange[lane] = l_sum;
        asm volatile("bar.sync %0, 64;" ::"r"(pair_barrier) : "memory");
        float total = l_sum;
        if (half == 0) {
            total += sum_exchange[lane];
            sum_exchange[lane] = total;
        }
        asm volatile("bar.sync %0, 64;" ::"r"(pair_barrier) : "memory");
        if (half == 1) total = sum_exchange[lane];
        if (args.row_max != nullptr || args.row_sum != nullptr) {
            // exact row maximum: the same two hand-overs with the f32 half-row maxima
            asm volatile("bar.sync %0, 64;" ::"r"(pair_barrier) : "memory");
            if (half == 1) sum_exchange[lane] = raw_max;
            asm volatile("bar.sync %0, 64;" ::"r"(pair_barrier) : "memory");
            if (half == 0) {
                const float row_raw_max = fmaxf(raw_max, sum_exchange[lane]);
                const int64_t b64 = item.batch, h64 = item.head, q64 = q_index;
                const bool any = !GENERAL || q_index < item.live_q;
                const bool inside = ok && q_index < args.seq_q;
                if (inside && args.row_max != nullptr)
                    args.row_max[b64 * args.max_stride[0] + h64 * args.max_stride[1] + q64 * args.max_stride[2]] = any ? row_raw_max * args.attn_scale : -INFINITY;
                if (inside && args.row_sum != nullptr)
                    args.row_sum[b64 * args.sum_stride[0] + h64 * args.sum_stride[1] + q64 * args.sum_stride[2]] = any ? sum_against<GENERAL>(total, m_ref, row_raw_max * scale) : 0.0f;
            }
        }
        // the hand-over words double as the next item's maxima: every read above must precede those writes
        asm volatile("bar.sync %0, 64;" ::"r"(pair_barrier) : "memory");
        const bool live = !GENERAL || q_index < item.live_q;
        const float inverse = live ? inverse_of<GENERAL>(total) : 0.0f;
        // the staging tile serves the query tiles in turn: A, B, the next item's A, ...
        {
            const uint32_t turn = 2 * n + x;
            if (ok) ok = mbar_wait(stage_free, (turn & 1) ^ 1, 232 + x);
        }
        uint8_t* o_row = generic_base + Smem::kStage + (D == 128 ? half * kHalfBytes : 0) + row * 128;  // this thread's output columns: 16-byte units from first_unit on
        const int first_unit = D == 128 ? 0 : half * 4;
#pragma unroll 1
        for (int c = 0; c < kColumns / 32; ++c) {
            uint32_t acc[32];
            tmem_load_32(tmem_o + c * 32, acc);
            tmem_load_wait();
            if (c == kColumns / 32 - 1) {
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(o_empty(x));
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                uint32_t w[4];
#pragma unroll
                for (int t = 0; t < 4; ++t)   // (selected, not multiplied: a dead row's accumulator may hold anything)
                    w[t] = live ? pack_pair<F16>(__uint_as_float(acc[u * 8 + 2 * t]) * inverse, __uint_as_float(acc[u * 8 + 2 * t + 1]) * inverse) : 0u;
                const int unit = first_unit + c * 4 + u;
                *reinterpret_cast<uint4*>(o_row + ((unit ^ (row & 7)) << 4)) = make_uint4(w[0], w[1], w[2], w[3]);
            }
        }
        fence_async_shared();
        __syncwarp();
        if (lane == 0) mbar_arrive(staged(x));
        if (args.stats != nullptr && ok && half == 0 && q_index < args.seq_q)
            args.stats[item.batch * args.stats_batch_stride + item.head * args.stats_head_stride + static_cast<int64_t>(q_index) * args.stats_row_stride] =
                live ? natural_log_sum<GENERAL>(args, m_ref, total) : -INFINITY;
        if (PADDED) ring_base += 2 * item.tiles;
        ++n;
        return true;  // also after a wait gave up: the two warps of a row pair must meet at the same barriers to the end
        });
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 17) {
        tc_fence_after();
        tmem_dealloc(tmem_base, 512);
    }
}

// ---- head dimension 128, few pairs: two SMs on a pair of query tiles ----------------------------
// A score tile lives in tensor memory from the product that writes it to the product that reads its probabilities: 512
// clocks of Q K^T, some 2600 of softmax and hand-overs, 512 of P V. With room for two tiles (two query tiles of one SM, each
// with a 128-column accumulator of its own) one tile leaves every ~1840 clocks whatever the order. Here an SM takes
// ONE query tile, whose accumulator leaves room for THREE score tiles of successive keys, and two SMs (a cluster) share
// the keys: rows 0-127 on CTA 0, rows 128-255 on CTA 1, one tcgen05.mma.cta_group::2 per step for both, each holding
// half of the K rows and half of the V columns, so that K and V are fetched and stored once per pair of query tiles as before.
//   warps 0-7, 8-15  softmax of the even and of the odd key tiles, two threads per query row
//   warp 16          TMA: own Q rows, own half of every K and V tile, in the order they are read: K0 K1 K2 V0 K3 V1 K4 ...
//   warp 17          of CTA 0 issues S(0) S(1) S(2) PV(0) S(3) PV(1) S(4) ..., on across items
//   warp 18          output tiles to global memory by TMA
// The reference maximum of a row goes from tile to tile: each group passes it on as soon as it has seen its own tile's
// maximum, before its exponentials. Tensor memory: S(t) and P(t) at 128 (t mod 3), O at 384.
constexpr int kDuoSlots = 6;
constexpr int kDuoBuffers = 3;
struct DuoSmem {
    static constexpr int kTile = kRows * 128 * 2;
    static constexpr int kSlot = kTile / 2;             // half a K or V tile
    static constexpr int kQ = 0;                        // this item's and the next one's
    static constexpr int kRing = 2 * kTile;
    static constexpr int kStage = kRing + kDuoSlots * kSlot;
    static constexpr int kMaxima = kStage + kTile;      // half-row maxima, bf16 (GENERAL: f32) [turn 2][group][quarter][half][lane]
    static constexpr int kReference = kMaxima + 4096;   // f32 [turn 2][group][half][quarter][lane]
    static constexpr int kSums = kReference + 4096;     // f32 {row sum, its reference, largest dot product} [group][half][row]
    static constexpr int kBarriers = kSums + 3 * 2048;
    // stage_free, staged, o_empty, sums_ready, sums_free, v_edge, edge_done, q_full[2], q_empty[2], kv_full[S],
    // kv_empty[S], s_full[3], p_full[3], pv_done[3], passed_on[group][half][quarter]
    static constexpr int kBarrierCount = 11 + 2 * kDuoSlots + 3 * kDuoBuffers + 16;
    static constexpr int kTotal = kBarriers + kBarrierCount * 8 + 16;
    static constexpr int kDynamic = kTotal + 1024;
};

__device__ __forceinline__ uint32_t duo_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void duo_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t address_in_first(uint32_t own_address) {
    uint32_t remote;
    asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(remote) : "r"(own_address));
    return remote;
}
__device__ __forceinline__ void arrive_in_cluster(uint32_t cluster_address) {
    // (for hand-overs of tensor memory alone, ordered by the tcgen05 fences. Released to the cluster, the arrival waits for every store
    // on its way, and a wait that acquires from the cluster takes 250 clocks even when it is over at once: only the tile whose V rows
    // are cleared in shared memory is handed over that way.)
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_address) : "memory");
}
__device__ __forceinline__ void commit_to_both(uint32_t bar) {
    const uint16_t both = 3;
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar), "h"(both) : "memory");
}
__device__ __forceinline__ void tma_load_4d_pair(uint32_t dst, const CUtensorMap* map, int c0, int c1, int c2, int c3, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.4d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];"
                 ::"r"(dst), "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(bar) : "memory");
}
__device__ __forceinline__ void duo_scores(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                 ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void duo_product(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
                 ::"r"(d), "r"(a), "l"(b), "r"(idesc), "r"(accumulate) : "memory");
}

// The key tiles of a cluster's work list, one after the other.
template <bool GENERAL>
struct TileCursor {
    PairWalker<2> walker;
    PairItem item;
    int j;        // key tile of the item
    uint32_t n;   // items before this one
    uint32_t t;   // key tiles before this one
    bool live;
    __device__ __forceinline__ void take(const SdpaUmmaArgs& args) {
        int bh, pair;
        live = walker.next(args, bh, pair);
        if (live) item = pair_item<GENERAL>(args, bh, pair);
        j = 0;
    }
    __device__ __forceinline__ void start(const SdpaUmmaArgs& args) {
        walker = PairWalker<2>();
        n = t = 0;
        take(args);
    }
    __device__ __forceinline__ bool last() const { return j + 1 == item.tiles; }
    __device__ __forceinline__ void step(const SdpaUmmaArgs& args) {
        ++t;
        if (++j == item.tiles) {
            ++n;
            take(args);
        }
    }
};
// The item's last key tile ends behind the batch's own length: V rows there are cleared.
__device__ __forceinline__ bool clears_v(const SdpaUmmaArgs& args, const PairItem& item) { return args.len_q != nullptr && item.tiles * kKeys > item.kv_len; }

template <bool F16, bool GENERAL>
__global__ void __launch_bounds__(kPairThreads, 1)
sdpa_umma_duo_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v,
                     const __grid_constant__ CUtensorMap map_o, SdpaUmmaArgs args) {
    using Smem = DuoSmem;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t* generic_base = smem_raw + (smem_base - smem_u32(smem_raw));
    const uint32_t bar_base = smem_base + Smem::kBarriers;
    const uint32_t stage_free = bar_base, staged = bar_base + 8, o_empty = bar_base + 16, sums_ready = bar_base + 24, sums_free = bar_base + 32, v_edge = bar_base + 40,
                   edge_done = bar_base + 48;
    auto q_full = [&](int i) { return bar_base + 8u * (7 + i); };
    auto q_empty = [&](int i) { return bar_base + 8u * (9 + i); };
    auto kv_full = [&](int s) { return bar_base + 8u * (11 + s); };
    auto kv_empty = [&](int s) { return bar_base + 8u * (11 + kDuoSlots + s); };
    auto s_full = [&](int b) { return bar_base + 8u * (11 + 2 * kDuoSlots + b); };
    auto p_full = [&](int b) { return bar_base + 8u * (11 + 2 * kDuoSlots + kDuoBuffers + b); };
    auto pv_done = [&](int b) { return bar_base + 8u * (11 + 2 * kDuoSlots + 2 * kDuoBuffers + b); };
    auto passed_on = [&](int group, int half, int quarter) { return bar_base + 8u * (11 + 2 * kDuoSlots + 3 * kDuoBuffers + group * 8 + half * 4 + quarter); };
    const uint32_t tmem_slot = bar_base + 8u * Smem::kBarrierCount;
    volatile uint32_t* tmem_slot_ptr = reinterpret_cast<volatile uint32_t*>(generic_base + Smem::kBarriers + 8 * Smem::kBarrierCount);
    volatile int* edge_slot = reinterpret_cast<volatile int*>(generic_base + Smem::kBarriers + 8 * Smem::kBarrierCount + 4);

    const int warp = uniform_warp_index(), lane = threadIdx.x & 31;
    const int rank = static_cast<int>(duo_rank());
    if (threadIdx.x == 0) {
        prefetch_tensormap(&map_q);
        prefetch_tensormap(&map_k);
        prefetch_tensormap(&map_v);
        prefetch_tensormap(&map_o);
        mbar_init(stage_free, 1);
        mbar_init(staged, 8);
        mbar_init(o_empty, 16);
        mbar_init(sums_ready, 8);
        mbar_init(sums_free, 8);
        mbar_init(v_edge, 1);
        mbar_init(edge_done, 8);
        for (int i = 0; i < 2; ++i) {
            mbar_init(q_full(i), 1);
            mbar_init(q_empty(i), 1);
        }
        for (int s = 0; s < kDuoSlots; ++s) {
            mbar_init(kv_full(s), 1);
            mbar_init(kv_empty(s), 1);
        }
        for (int b = 0; b < kDuoBuffers; ++b) {
            mbar_init(s_full(b), 1);
            mbar_init(p_full(b), 16);
            mbar_init(pv_done(b), 1);
        }
        for (int i = 0; i < 16; ++i) mbar_init(passed_on(0, 0, 0) + 8u * i, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 17) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tmem_slot), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
        tc_fence_before();
    }
    __syncthreads();
    duo_sync();   // both CTAs' barriers exist before either touches the other's
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot_ptr;
    chain_wait();
    chain_release();

    if (warp == 16) {
        const bool leader = elect_one();
        const uint32_t counted_on = address_in_first(bar_base);   // CTA 0's barriers count both CTAs' bytes
        TileCursor<GENERAL> k, v;
        k.start(args);
        v.start(args);
        int slot = 0;
        uint32_t phase = 1, edges = 0;
        bool ok = true;
        auto next_slot = [&] { if (++slot == kDuoSlots) { slot = 0; phase ^= 1; } };
        auto put_k = [&] {
            if (!k.live || !ok) return;
            if (k.j == 0) {
                const int buffer = k.n & 1;
                ok = mbar_wait_warp(q_empty(buffer), ((k.n >> 1) & 1) ^ 1, 240);
                if (leader && ok) {
                    if (rank == 0) mbar_expect_tx(q_full(buffer), 2 * Smem::kTile);
                    for (int h = 0; h < 2; ++h)
                        tma_load_4d_pair(smem_base + Smem::kQ + buffer * Smem::kTile + h * kHalfBytes, &map_q, 64 * h, (k.item.q_tile_a + rank) * kRows, k.item.head, k.item.batch,
                                         counted_on + (q_full(buffer) - bar_base));
                }
            }
            if (ok) ok = mbar_wait_warp(kv_empty(slot), phase, 241);
            if (leader && ok) {
                if (rank == 0) mbar_expect_tx(kv_full(slot), 2 * Smem::kSlot);
                for (int h = 0; h < 2; ++h)
                    tma_load_4d_pair(smem_base + Smem::kRing + slot * Smem::kSlot + h * (Smem::kSlot / 2), &map_k, 64 * h, k.j * kKeys + rank * 64, k.item.kv_head, k.item.batch,
                                     counted_on + (kv_full(slot) - bar_base));
            }
            __syncwarp();
            next_slot();
            k.step(args);
        };
        for (int i = 0; i < kDuoBuffers; ++i) put_k();
        while (v.live && ok) {
            const bool edge = GENERAL && v.last() && clears_v(args, v.item);
            ok = mbar_wait_warp(kv_empty(slot), phase, 242);
            // (a tile whose end is cleared is counted on a barrier of its own CTA, where the clearing warps wait for it)
            if (edge && ok) ok = mbar_wait_warp(edge_done, (edges & 1) ^ 1, 243);
            if (leader && ok) {
                const uint32_t dst = smem_base + Smem::kRing + slot * Smem::kSlot;
                if (edge) {
                    *edge_slot = slot;
                    if (rank == 0) mbar_arrive(kv_full(slot));
                    mbar_expect_tx(v_edge, Smem::kSlot);
                    tma_load_4d(dst, &map_v, 64 * rank, v.j * kKeys, v.item.kv_head, v.item.batch, v_edge);
                } else {
                    if (rank == 0) mbar_expect_tx(kv_full(slot), 2 * Smem::kSlot);
                    tma_load_4d_pair(dst, &map_v, 64 * rank, v.j * kKeys, v.item.kv_head, v.item.batch, counted_on + (kv_full(slot) - bar_base));
                }
            }
            __syncwarp();
            edges += edge ? 1 : 0;
            next_slot();
            v.step(args);
            put_k();
        }
    } else if (warp == 17) {
        if (rank == 0) {
            const bool leader = elect_one();
            constexpr uint32_t kFormats = (1u << 4) | (F16 ? 0u : (1u << 7) | (1u << 10)) | (static_cast<uint32_t>(2 * kRows >> 4) << 24);
            const uint32_t idesc_qk = kFormats | (static_cast<uint32_t>(kKeys >> 3) << 17) | args.negate_q;
            constexpr uint32_t idesc_pv = kFormats | (static_cast<uint32_t>(128 >> 3) << 17) | (1u << 16);   // (V is read MN-major)
            constexpr uint32_t kDescHi = smem_desc_hi(1024);
            const uint32_t tmem_u = __shfl_sync(0xffffffffu, tmem_base, 0);
            TileCursor<GENERAL> s, p;
            s.start(args);
            p.start(args);
            int slot = 0;
            uint32_t phase = 0;
            bool ok = true;
            auto next_slot = [&] { if (++slot == kDuoSlots) { slot = 0; phase ^= 1; } };
            auto put_scores = [&] {
                if (!s.live || !ok) return;
                const int q = s.n & 1, b = static_cast<int>(s.t % kDuoBuffers);
                if (s.j == 0) ok = mbar_wait_warp(q_full(q), (s.n >> 1) & 1, 244);
                if (ok) ok = mbar_wait_warp(kv_full(slot), phase, 245);
                tc_fence_after();
                if (leader && ok) {
                    const uint32_t q_lo = smem_desc_lo(smem_base + Smem::kQ + q * Smem::kTile, 16), k_lo = smem_desc_lo(smem_base + Smem::kRing + slot * Smem::kSlot, 16);
#pragma unroll
                    for (int k = 0; k < 8; ++k)
                        duo_scores(tmem_u + b * 128, desc_words(q_lo + (((k >> 2) * kHalfBytes + (k & 3) * 32) >> 4), kDescHi),
                                   desc_words(k_lo + (((k >> 2) * (Smem::kSlot / 2) + (k & 3) * 32) >> 4), kDescHi), idesc_qk, k != 0 ? 1u : 0u);
                    commit_to_both(s_full(b));
                    commit_to_both(kv_empty(slot));
                    if (s.last()) commit_to_both(q_empty(q));
                }
                __syncwarp();
                next_slot();
                s.step(args);
            };
            for (int i = 0; i < kDuoBuffers; ++i) put_scores();
            while (p.live && ok) {
                const int b = static_cast<int>(p.t % kDuoBuffers);
                if (p.j == 0) ok = mbar_wait_warp(o_empty, (p.n & 1) ^ 1, 246);
                if (ok) ok = mbar_wait_warp(kv_full(slot), phase, 247);
                if (GENERAL && p.last() && clears_v(args, p.item)) {   // (V rows that both CTAs' warps have cleared)
                    if (ok) ok = mbar_wait_warp_cluster(p_full(b), (p.t / kDuoBuffers) & 1, 248);
                } else {
                    if (ok) ok = mbar_wait_warp(p_full(b), (p.t / kDuoBuffers) & 1, 248);
                }
                tc_fence_after();
                if (leader && ok) {
                    const uint32_t v_lo = smem_desc_lo(smem_base + Smem::kRing + slot * Smem::kSlot, kHalfBytes), p_tmem = tmem_u + b * 128;
#pragma unroll
                    for (int k = 0; k < 8; ++k) {
                        const uint32_t p_at = p_tmem + (k >> 2) * 64 + (k & 3) * kProbabilityColumns<GENERAL>;
                        duo_product(tmem_u + 384, p_at, desc_words(v_lo + ((k * 2048) >> 4), kDescHi), idesc_pv, (p.j | k) != 0 ? 1u : 0u);
                        if constexpr (GENERAL) duo_product(tmem_u + 384, p_at + 8, desc_words(v_lo + ((k * 2048) >> 4), kDescHi), idesc_pv, 1u);
                    }
                    commit_to_both(pv_done(b));
                    commit_to_both(kv_empty(slot));
                }
                __syncwarp();
                next_slot();
                p.step(args);
                put_scores();   // (into the buffer just read: the products of one thread run in order)
            }
        }
    } else if (warp == 18) {
        const bool leader = elect_one();
        uint32_t n = 0;
        bool ok = true;
        for_each_pair_item<2, false>(args, nullptr, [&](int bh, int pair) {
            const PairItem item = pair_item<GENERAL>(args, bh, pair);
            if (ok) ok = mbar_wait_warp(staged, n & 1, 249);
            if (leader) {
                const int row = (item.q_tile_a + rank) * kRows;
                if (ok && g_device_status == 0 && row < args.seq_q)
                    for (int h = 0; h < 2; ++h) tma_store_4d(&map_o, smem_base + Smem::kStage + h * kHalfBytes, 64 * h, row, item.head, item.batch);
                tma_store_commit();
                tma_store_wait_read<0>();
                mbar_arrive(stage_free);
            }
            __syncwarp();
            ++n;
            return true;
        });
        if (leader) tma_store_wait_all();
    } else {
        const int group = warp >> 3, half = (warp >> 2) & 1, quarter = warp & 3;
        const int row = quarter * 32 + lane;
        const uint32_t lane_base = static_cast<uint32_t>(quarter * 32) << 16;
        const uint32_t tmem_o = tmem_base + lane_base + 384 + half * 64;
        const float scale = args.scale_log2;
        const uint64_t scale2 = pack2(scale, scale);
        const int pair_barrier = 1 + group * 4 + quarter;   // the 64 threads of this group that share these 32 rows
        uint16_t* maxima = reinterpret_cast<uint16_t*>(generic_base + Smem::kMaxima) + (group * 4 + quarter) * 64 + lane;          // + turn * 512 + half * 32
        float* reference = reinterpret_cast<float*>(generic_base + Smem::kReference) + (half * 4 + quarter) * 32 + lane;           // + turn * 512 + group * 256
        float* sums_of = reinterpret_cast<float*>(generic_base + Smem::kSums) + row;   // + 512 * {sum, reference, largest} + (group * 2 + half) * 128
        const uint32_t p_full_first = address_in_first(p_full(0)), o_empty_first = address_in_first(o_empty);
        uint32_t n = 0, t0 = 0, edges = 0;
        uint32_t mine_done = 0;   // key tiles this group has finished (parity of its maxima and references)
        bool ok = true;
        for_each_pair_item<2, false>(args, nullptr, [&](int bh, int pair) {
            const PairItem item = pair_item<GENERAL>(args, bh, pair);
            const int q_tile = item.q_tile_a + rank, q_index = q_tile * kRows + row;
            const bool idle_tile = q_tile * kRows >= item.live_q;   // no row of this CTA's has keys
            float m_ref = -INFINITY, l_sum = 0.0f, raw_max = -INFINITY;
            // The reference after key tile t, as the other group passed it on. That group's own count of tiles gives buffer and phase:
            // tiles of its parity before t.
            auto passed = [&](uint32_t t) {
                const uint32_t turn = t >> 1;   // (tile t is the turn-th of its group)
                if (ok) ok = mbar_wait(passed_on(group ^ 1, half, quarter), turn & 1, 250);
                return reference[(turn & 1) * 512 + (group ^ 1) * 256];
            };
            for (int j = static_cast<int>((t0 ^ group) & 1); j < item.tiles; j += 2, ++mine_done) {
                const uint32_t t = t0 + j;
                const int b = static_cast<int>(t % kDuoBuffers);
                const uint32_t tmem_s = tmem_base + lane_base + b * 128 + half * 64;
                // (S(t) follows PV(t - 3): what this tile's turn of the buffers held before has been read, and no barrier below is more than one phase behind)
                if (ok) ok = mbar_wait(s_full(b), (t / kDuoBuffers) & 1, 251);
                tc_fence_after();
                const bool empty = idle_tile || (args.causal && j > q_tile);   // nothing to see for any row: all probabilities are zero
                const int last_key = !GENERAL ? q_index : (args.causal ? min(q_index, item.kv_len - 1) : item.kv_len - 1);
                const int limit = last_key - j * kKeys - half * 64;
                const bool diagonal = (args.causal && j == q_tile) || (GENERAL && (j + 1) * kKeys > item.kv_len);
                // The tile's maximum first, then the reference, then the exponentials: nothing is formed twice. (The scores are read
                // twice, which costs next to nothing; 64 of them held in registers would spill.)
                float mine = -INFINITY;
                auto masked = [&](uint32_t (&raw)[16], int c) {
                    if (diagonal) {
#pragma unroll
                        for (int e = 0; e < 16; ++e)
                            if (c * 16 + e > limit) raw[e] = 0xff800000u;  // -inf
                    }
                };
                if (!empty) {
                    uint32_t raw[4][16];
                    tmem_load_16(tmem_s, raw[0]);
                    tmem_load_16(tmem_s + 16, raw[1]);
#pragma unroll
                    for (int c = 0; c < 4; c += 2) {
                        tmem_load_wait_for(raw[c]);
                        tmem_load_wait_for(raw[c + 1]);
                        if (c < 2) {
                            tmem_load_16(tmem_s + 32, raw[2]);
                            tmem_load_16(tmem_s + 48, raw[3]);
                        }
                        masked(raw[c], c);
                        masked(raw[c + 1], c + 1);
                        mine = max_of_16(raw[c + 1], max_of_16(raw[c], mine));
                    }
                }
                raw_max = fmaxf(raw_max, mine);
                // Half-row maxima as bf16 rounded towards +inf: any reference not below the true maximum by more than the threshold
                // serves, and both threads must arrive at the same value. (Two buffers: the other warp may still be reading the
                // last tile's when this one writes.)
                const uint32_t turn = mine_done & 1;
                float tile_max;
                if constexpr (GENERAL) {   // (exact: see the kernel above)
                    float* exact = reinterpret_cast<float*>(generic_base + Smem::kMaxima) + (group * 4 + quarter) * 64 + lane;
                    exact[turn * 512 + half * 32] = mine;
                    asm volatile("bar.sync %0, 64;" ::"r"(pair_barrier) : "memory");
                    tile_max = fmaxf(mine, exact[turn * 512 + (half ^ 1) * 32]) * scale;
                } else {
                    const uint32_t mine_up = round_up<16>(mine);
                    maxima[turn * 512 + half * 32] = static_cast<uint16_t>(mine_up >> 16);
                    asm volatile("bar.sync %0, 64;" ::"r"(pair_barrier) : "memory");
                    tile_max = fmaxf(__uint_as_float(mine_up), __uint_as_float(static_cast<uint32_t>(maxima[turn * 512 + (half ^ 1) * 32]) << 16)) * scale;
                }
                float before = t > 0 ? passed(t - 1) : -INFINITY;   // (at an item's start for the order alone: the other group has taken what this one passed on last)
                if (j == 0) before = -INFINITY;
                // raise the reference only when it would grow by more than the threshold (or on the first tile)
                const bool raise = __any_sync(0xffffffffu, tile_max > before + kRescaleThreshold) != 0;
                const float m_new = raise ? fmaxf(before, tile_max) : before;
                reference[turn * 512 + group * 256] = m_new;
                __syncwarp();
                if (lane == 0) mbar_arrive(passed_on(group, half, quarter));
                if (__any_sync(0xffffffffu, m_new != m_ref)) {
                    l_sum *= m_ref == -INFINITY ? 0.0f : ex2_fast(m_ref - m_new);
                    m_ref = m_new;
                }
                uint64_t sums[2] = {0, 0};
                if (!empty) {
                    // (probabilities go over columns whose scores have been read: 8 columns for every 16, or all 16)
                    const uint64_t bias2 = pack2(bias_of<GENERAL>(m_ref), bias_of<GENERAL>(m_ref));
                    uint32_t raw[4][16];
                    tmem_load_16(tmem_s, raw[0]);
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        tmem_load_wait_for(raw[c]);
                        if (c < 3) tmem_load_16(tmem_s + (c + 1) * 16, raw[c + 1]);
                        masked(raw[c], c);
                        put_probabilities<F16, GENERAL>(raw[c], scale2, bias2, sums, tmem_s + c * kProbabilityColumns<GENERAL>);
                    }
                } else {
                    const uint32_t zeros[8] = {};
#pragma unroll
                    for (int c = 0; c < kProbabilityColumns<GENERAL> / 2; ++c) tmem_store_8(tmem_s + c * 8, zeros);
                }
                {
                    float lo, hi;
                    unpack2(add2(sums[0], sums[1]), lo, hi);
                    l_sum += lo + hi;
                }
                if (raise && j > 0) {
                    // O holds P V up to the tile before once that product is done; this tile's waits for these probabilities.
                    const float alpha = before == -INFINITY ? 0.0f : ex2_fast(before - m_new);
                    if (ok) ok = mbar_wait(pv_done((t - 1) % kDuoBuffers), ((t - 1) / kDuoBuffers) & 1, 252);
                    tc_fence_after();
#pragma unroll 1
                    for (int c = 0; c < 4; ++c) {
                        uint32_t acc[16];
                        tmem_load_16(tmem_o + c * 16, acc);
                        tmem_load_wait_for(acc);
#pragma unroll
                        for (int e = 0; e < 16; ++e) acc[e] = __float_as_uint(__uint_as_float(acc[e]) * alpha);
                        tmem_store_16(tmem_o + c * 16, acc);
                    }
                }
                const bool cleared = GENERAL && half == 0 && j + 1 == item.tiles && clears_v(args, item);
                if (cleared) {
                    // V rows past the batch's length are not this sequence's: this CTA's channels of them, a row per thread
                    if (ok) ok = mbar_wait(v_edge, edges & 1, 253);
                    if (j * kKeys + row >= item.kv_len) {
                        uint8_t* v_row = generic_base + Smem::kRing + *edge_slot * Smem::kSlot + row * 128;
#pragma unroll
                        for (int u = 0; u < 8; ++u) *reinterpret_cast<uint4*>(v_row + u * 16) = make_uint4(0, 0, 0, 0);
                    }
                    fence_async_shared();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(edge_done);
                }
                tmem_store_wait();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) {
                    if (cleared) mbar_arrive_cluster_release(p_full_first + 8u * b);
                    else arrive_in_cluster(p_full_first + 8u * b);
                }
            }
            const uint32_t last = t0 + item.tiles - 1;
            if (GENERAL && clears_v(args, item)) {
                // (the group that does not clear waits and arrives as well: a barrier's phases are told apart by their parity, so nobody may
                // be more than one behind or ahead)
                if (half == 0 && (last & 1) != static_cast<uint32_t>(group)) {
                    if (ok) ok = mbar_wait(v_edge, edges & 1, 258);
                    __syncwarp();
                    if (lane == 0) mbar_arrive(edge_done);
                }
                ++edges;
            }
            // ---- the item's end: the group without the last tile leaves its sums, the other one finishes the rows ----
            t0 += item.tiles;
            float* own = sums_of + (group * 2 + half) * 128;
            if (ok) ok = mbar_wait(sums_free, (n & 1) ^ 1, 254);   // (the last item's sums have been read)
            if ((last & 1) != static_cast<uint32_t>(group)) {
                own[0] = l_sum;
                own[512] = m_ref;
                own[1024] = raw_max;
                __syncwarp();
                if (lane == 0) mbar_arrive(sums_ready);
            } else {
                if (ok) ok = mbar_wait(sums_ready, n & 1, 255);
                own[0] = l_sum;
                own[1024] = raw_max;
                asm volatile("bar.sync %0, 64;" ::"r"(pair_barrier) : "memory");
                float total = sums_of[group * 256] + sums_of[group * 256 + 128], row_raw_max = fmaxf(sums_of[group * 256 + 1024], sums_of[group * 256 + 128 + 1024]);
                const float other_ref = sums_of[512 + (group ^ 1) * 256];   // (both halves of a row know the same reference)
                if (other_ref != -INFINITY) {
                    total += (sums_of[(group ^ 1) * 256] + sums_of[(group ^ 1) * 256 + 128]) * ex2_fast(other_ref - m_ref);
                    row_raw_max = fmaxf(row_raw_max, fmaxf(sums_of[(group ^ 1) * 256 + 1024], sums_of[(group ^ 1) * 256 + 128 + 1024]));
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(sums_free);
                const bool live = !GENERAL ? true : q_index < item.live_q;
                if (half == 0 && ok && q_index < args.seq_q) {
                    const int64_t b64 = item.batch, h64 = item.head, q64 = q_index;
                    if (args.row_max != nullptr)
                        args.row_max[b64 * args.max_stride[0] + h64 * args.max_stride[1] + q64 * args.max_stride[2]] = live ? row_raw_max * args.attn_scale : -INFINITY;
                    if (args.row_sum != nullptr)
                        args.row_sum[b64 * args.sum_stride[0] + h64 * args.sum_stride[1] + q64 * args.sum_stride[2]] = live ? sum_against<GENERAL>(total, m_ref, row_raw_max * scale) : 0.0f;
                    if (args.stats != nullptr)
                        args.stats[b64 * args.stats_batch_stride + h64 * args.stats_head_stride + q64 * args.stats_row_stride] =
                            live ? natural_log_sum<GENERAL>(args, m_ref, total) : -INFINITY;
                }
                const float inverse = live ? inverse_of<GENERAL>(total) : 0.0f;
                if (ok) ok = mbar_wait(stage_free, (n & 1) ^ 1, 256);
                if (ok) ok = mbar_wait(pv_done(last % kDuoBuffers), (last / kDuoBuffers) & 1, 257);
                tc_fence_after();
                uint8_t* o_row = generic_base + Smem::kStage + half * kHalfBytes + row * 128;
#pragma unroll 1
                for (int c = 0; c < 2; ++c) {
                    uint32_t acc[32];
                    tmem_load_32(tmem_o + c * 32, acc);
                    tmem_load_wait();
                    if (c == 1) {
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) arrive_in_cluster(o_empty_first);
                    }
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        uint32_t w[4];
#pragma unroll
                        for (int i = 0; i < 4; ++i)   // (selected, not multiplied: a dead row's accumulator may hold anything)
                            w[i] = live ? pack_pair<F16>(__uint_as_float(acc[u * 8 + 2 * i]) * inverse, __uint_as_float(acc[u * 8 + 2 * i + 1]) * inverse) : 0u;
                        *reinterpret_cast<uint4*>(o_row + (((c * 4 + u) ^ (row & 7)) << 4)) = make_uint4(w[0], w[1], w[2], w[3]);
                    }
                }
                fence_async_shared();
                __syncwarp();
                if (lane == 0) mbar_arrive(staged);
            }
            ++n;
            return true;  // also after a wait gave up: the warps of a row must meet at the same barriers to the end
        });
    }

    tc_fence_before();
    __syncthreads();
    duo_sync();   // no CTA leaves while the other may still signal its barriers or read its operands
    if (warp == 17) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
    }
}

// Channel-contiguous [B, H, S, D] whose rows TMA can read: every other stride a positive multiple of 16 bytes.
bool rows_for_tma(const dfgpu_tensor& t) {
    if (t.rank != 4 || t.stride[3] != 1) return false;
    for (int i = 0; i < 3; ++i)
        if (t.dim[i] != 1 && (t.stride[i] <= 0 || t.stride[i] % 8 != 0 || t.stride[i] >= (1ll << 38))) return false;
    return t.dim[0] < (1ll << 31) && t.dim[1] < (1ll << 31) && t.dim[2] < (1ll << 30);
}

int sdpa_map(CUtensorMap* map, const dfgpu_tensor& t, const void* data, uint32_t rows, const char* what) {
    uint64_t dims[4] = {static_cast<uint64_t>(t.dim[3]), static_cast<uint64_t>(t.dim[2]), static_cast<uint64_t>(t.dim[1]), static_cast<uint64_t>(t.dim[0])};
    uint64_t strides[3];
    for (int i = 0; i < 3; ++i) strides[i] = static_cast<uint64_t>(t.dim[2 - i] == 1 ? t.dim[3] : t.stride[2 - i]) * 2;   // (an axis of one position has no stride to mind)
    uint32_t box[4] = {64, rows, 1, 1};
    return make_map(map, data, 4, dims, strides, box, what);
}

template <int D, bool F16, bool GENERAL, bool PADDED>
int launch_pair(const CUtensorMap& map_q, const CUtensorMap& map_k, const CUtensorMap& map_v, const CUtensorMap& map_o, const SdpaUmmaArgs& args, unsigned grid, cudaStream_t stream) {
    cudaError_t error = cudaFuncSetAttribute(sdpa_umma_pair_kernel<D, F16, GENERAL, PADDED>, cudaFuncAttributeMaxDynamicSharedMemorySize, PairSmem<D>::kDynamic);
    if (error != cudaSuccess) return fail(kExecutionFailed, "SDPA: cannot reserve %d bytes of shared memory: %s", PairSmem<D>::kDynamic, cudaGetErrorString(error));
    launch_chained(sdpa_umma_pair_kernel<D, F16, GENERAL, PADDED>, dim3(grid), dim3(kPairThreads), PairSmem<D>::kDynamic, stream, map_q, map_k, map_v, map_o, args);
    return check_launch("SDPA (tcgen05, two query tiles per CTA)");
}
template <bool F16, bool GENERAL>
int launch_duo(const CUtensorMap& map_q, const CUtensorMap& map_k, const CUtensorMap& map_v, const CUtensorMap& map_o, const SdpaUmmaArgs& args, unsigned clusters, cudaStream_t stream) {
    cudaError_t error = cudaFuncSetAttribute(sdpa_umma_duo_kernel<F16, GENERAL>, cudaFuncAttributeMaxDynamicSharedMemorySize, DuoSmem::kDynamic);
    if (error != cudaSuccess) return fail(kExecutionFailed, "SDPA: cannot reserve %d bytes of shared memory: %s", DuoSmem::kDynamic, cudaGetErrorString(error));
    error = launch_chained_cluster(sdpa_umma_duo_kernel<F16, GENERAL>, dim3(2 * clusters), dim3(kPairThreads), 2u, static_cast<size_t>(DuoSmem::kDynamic), stream, map_q, map_k, map_v, map_o, args);
    if (error != cudaSuccess) return fail(kExecutionFailed, "SDPA: launch failed: %s", cudaGetErrorString(error));
    return check_launch("SDPA (tcgen05, two SMs per pair of query tiles)");
}
template <int D, bool F16>
int launch_general(bool duo, const CUtensorMap& map_q, const CUtensorMap& map_k, const CUtensorMap& map_v, const CUtensorMap& map_o, const SdpaUmmaArgs& args, unsigned grid, cudaStream_t stream) {
    if constexpr (D == 128)
        if (duo) return launch_duo<F16, true>(map_q, map_k, map_v, map_o, args, grid, stream);
    return args.len_q != nullptr ? launch_pair<D, F16, true, true>(map_q, map_k, map_v, map_o, args, grid, stream)
                                 : launch_pair<D, F16, true, false>(map_q, map_k, map_v, map_o, args, grid, stream);
}

bool packed_rows(const dfgpu_tensor& t) {
    return t.stride[3] == 1 && t.stride[2] == t.dim[3] && t.stride[1] == t.dim[2] * t.stride[2] && t.stride[0] == t.dim[1] * t.stride[1];
}
// Whole 128-row tiles of packed bf16 rows of 128, no padding, a causal mask on square scores only: P V on P rounded to bf16.
bool plain_tiles(const dfgpu_sdpa_params& p) {
    const int64_t sq = p.q.dim[2], skv = p.k.dim[2];
    return p.q.dtype == DFGPU_BF16 && p.q.dim[3] == 128 && !p.padding_mask && sq % kRows == 0 && skv % kKeys == 0 && (!p.has_right_bound || sq == skv) &&
           packed_rows(p.q) && packed_rows(p.k) && packed_rows(p.v) && packed_rows(p.o) &&
           ((p.max.rank == 0 && p.sum_exp.rank == 0) || (sq % (2 * kRows) == 0 && p.attn_scale > 0.0f)) && p.q.dim[0] * p.q.dim[1] <= 65535;
}

}  // namespace

bool sdpa_umma_supported(const dfgpu_sdpa_params& p) {
    if (p.q.dtype != DFGPU_BF16 && p.q.dtype != DFGPU_F16) return false;
    if (p.k.dtype != p.q.dtype || p.v.dtype != p.q.dtype || p.o.dtype != p.q.dtype) return false;
    if (p.q.rank != 4 || p.k.rank != 4 || p.v.rank != 4 || p.o.rank != 4) return false;
    const int64_t d = p.q.dim[3];
    if ((d != 64 && d != 128) || p.v.dim[3] != d || p.k.dim[3] != d || p.o.dim[3] != d) return false;
    if (p.page_table_k.rank || p.page_table_v.rank || p.has_left_bound || p.bottom_right) return false;
    if (!rows_for_tma(p.q) || !rows_for_tma(p.k) || !rows_for_tma(p.v) || !rows_for_tma(p.o)) return false;
    const int64_t sq = p.q.dim[2], skv = p.k.dim[2];
    if (p.s_kv != skv || p.v.dim[2] != skv || p.k.dim[1] != p.v.dim[1]) return false;
    if (p.has_right_bound && p.right_bound != 0) return false;  // causal, top-left aligned
    if (!(p.attn_scale > -INFINITY && p.attn_scale < INFINITY)) return false;
    for (const dfgpu_tensor* row : {&p.stats, &p.max, &p.sum_exp})
        if (row->rank && row->dtype != DFGPU_F32) return false;
    return p.q.dim[0] * p.q.dim[1] * ((sq + 2 * kRows - 1) / (2 * kRows)) < (1ll << 30);
}

int launch_sdpa_umma(const dfgpu_sdpa_params& p, void* const* tensors, cudaStream_t stream) {
    for (int i = 0; i < 4; ++i)
        if ((reinterpret_cast<uintptr_t>(tensors[i]) & 15u) != 0) return fail(kInvalidArgument, "SDPA: the tcgen05 kernel needs 16-byte aligned Q, K, V and O");
    // One SM or two per pair of query tiles: the longest list of key tiles any of them walks, times what a tile step costs (two
    // tiles in 3670 clocks on one SM, one in 1620 on each of two; the latter count for 12 % more, since they draw more and a chip that is
    // full has to lower its clocks), and 4500 clocks a pair. (3670 is from before the hand-over in halves, which takes 1.5 to 7 % off it; a padded step is
    // 4400, and lengths are not looked at: 4 x 16 x 569 queries on up to 370 keys are 17.3 us on one SM each and 21.6 on the two they get.) A
    // causal pair's last tile is all masked for the first query tile, which one SM skips; so it does a second query tile that does not exist.
    //   64 pairs, 2048 causal: 35 us on one SM each, 21 on two. 96: 35 / 21. 16 x 2171 causal: 44 / 33. 8 x 32 x 2048 causal: 283 / 333 (329 / 351
    //   once the power limit holds). 192 x 1538 queries on 190 keys: 81 / 107.
    const int64_t pairs = (p.q.dim[2] + 2 * kRows - 1) / (2 * kRows), heads = p.q.dim[0] * p.q.dim[1], kv_tiles = (p.k.dim[2] + kKeys - 1) / kKeys;
    int64_t longest = 0, all = 0;
    for (int64_t i = 0; i < pairs; ++i) {
        const int64_t tiles = p.has_right_bound ? std::min(kv_tiles, 2 * i + 2) : kv_tiles;
        longest = std::max(longest, tiles);
        all += tiles * heads;
    }
    auto clocks = [&](int64_t places, double step) {
        constexpr double kPerPair = 4500.0;
        if (p.has_right_bound) return std::max(longest * step + kPerPair, (all * step + pairs * heads * kPerPair) / places);
        return static_cast<double>((pairs * heads + places - 1) / places) * (kv_tiles * step + kPerPair);
    };
    const double one = clocks(sm_count(), 3670.0 * (p.has_right_bound ? 0.94 : 1.0) * (p.q.dim[2] <= kRows ? 0.75 : 1.0)), two = clocks(sm_count() / 2, 1620.0 * 1.12);
    const bool duo = p.q.dim[3] == 128 && two < one;
    CUtensorMap map_q, map_k, map_v, map_o;
    int status = sdpa_map(&map_q, p.q, tensors[0], kRows, "SDPA Q");
    if (!status) status = sdpa_map(&map_k, p.k, tensors[1], duo ? kKeys / 2 : kKeys, "SDPA K");
    if (!status) status = sdpa_map(&map_v, p.v, tensors[2], kRows, "SDPA V");
    if (!status) status = sdpa_map(&map_o, p.o, tensors[3], kRows, "SDPA O");
    if (status) return status;
    SdpaUmmaArgs args{};
    args.heads_q = static_cast<int>(p.q.dim[1]);
    args.heads_kv = static_cast<int>(p.k.dim[1]);
    args.seq_q = static_cast<int>(p.q.dim[2]);
    args.seq_kv = static_cast<int>(p.k.dim[2]);
    args.pairs = static_cast<int>(pairs);
    args.batch_heads = static_cast<int>(p.q.dim[0] * p.q.dim[1]);
    args.causal = p.has_right_bound ? 1 : 0;
    // (a scale of zero weighs every key alike; the smallest normal one does too, and keeps scale * -inf at -inf)
    args.attn_scale = std::max(std::fabs(p.attn_scale), 1e-37f);
    args.scale_log2 = args.attn_scale * 1.4426950408889634f;
    const double to_natural = static_cast<double>(args.attn_scale) / args.scale_log2;
    args.to_natural[0] = static_cast<float>(to_natural);
    args.to_natural[1] = static_cast<float>(to_natural - args.to_natural[0]);
    args.negate_q = p.attn_scale < 0.0f ? 1u << 13 : 0u;
    if (p.padding_mask) {
        args.len_q = static_cast<const int32_t*>(tensors[7]);
        args.len_kv = static_cast<const int32_t*>(tensors[8]);
        args.len_q_stride = p.seq_q.stride[0];
        args.len_kv_stride = p.seq_kv.stride[0];
    }
    if (p.stats.rank) {
        args.stats = static_cast<float*>(tensors[4]);
        args.stats_batch_stride = p.stats.stride[0];
        args.stats_head_stride = p.stats.stride[1];
        args.stats_row_stride = p.stats.stride[2];
    }
    args.row_max = p.max.rank ? static_cast<float*>(tensors[5]) : nullptr;
    args.row_sum = p.sum_exp.rank ? static_cast<float*>(tensors[6]) : nullptr;
    for (int i = 0; i < 3; ++i) {
        args.max_stride[i] = p.max.rank ? p.max.stride[i] : 0;
        args.sum_stride[i] = p.sum_exp.rank ? p.sum_exp.stride[i] : 0;
    }
    // persistent: one CTA (or cluster of two) per SM (or two) over the work list (see PairWalker)
    const int places = duo ? sm_count() / 2 : sm_count();
    const int64_t single = pairs * heads;
    args.order = !args.causal || single <= places ? kAsStored : (duo ? kHeaviestFirst : kHeavyWithLight);   // (the third order in the one-SM kernel cost it 1.4 %)
    // By length where lengths can differ: with one key tile all pairs are alike, and with one pair a sequence that sees all keys nearly so up to
    // three tiles. Making the list costs each CTA 0.3 to 2 us there (5 x 32 x 108 causal 16.3 us without, 18.5 with; 15 x 2 x 2326 on 101 keys 21.0 and
    // 22.8; 32 x 8 x 101 on 290 16.3 and 17.1). From two tiles on it gains (20 x 32 x 298 on 146 keys 102 and 85; 29 x 8 x 154 causal 16.9 and 15.2).
    // CTAs that run side by side then read different heads' K and V: only where all of them stay in the L2 cache. An entry of the list is a
    // byte, 256 of them fit behind the barriers.
    const int64_t kv_bytes = p.k.dim[0] * p.k.dim[1] * p.k.dim[2] * p.k.dim[3] * 4;
    const bool uneven = kv_tiles > 1 && (pairs > 1 || args.causal || kv_tiles > 3);
    if (!duo && p.padding_mask && single > places && uneven && p.q.dim[0] * pairs <= PairSmem<128>::kMostPairs && kv_bytes <= (64 << 20)) args.order = kLongestFirst;
    const int64_t units = args.order == kHeavyWithLight ? (pairs + 1) / 2 * heads : single;
    const unsigned grid = static_cast<unsigned>(std::min<int64_t>(units, places));
    if (plain_tiles(p)) return duo ? launch_duo<false, false>(map_q, map_k, map_v, map_o, args, grid, stream) : launch_pair<128, false, false, false>(map_q, map_k, map_v, map_o, args, grid, stream);
    const bool f16 = p.q.dtype == DFGPU_F16;
    if (p.q.dim[3] == 64) return f16 ? launch_general<64, true>(duo, map_q, map_k, map_v, map_o, args, grid, stream) : launch_general<64, false>(duo, map_q, map_k, map_v, map_o, args, grid, stream);
    return f16 ? launch_general<128, true>(duo, map_q, map_k, map_v, map_o, args, grid, stream) : launch_general<128, false>(duo, map_q, map_k, map_v, map_o, args, grid, stream);
}

int sdpa_umma_device_status(int* status) { return read_and_clear_device_status(status); }

}  // namespace dfgpu
