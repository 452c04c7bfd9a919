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
// probability times an infinity in the padding would be NaN), and rows past SEQ_LEN_Q store 0 and -inf.
#include <algorithm>
#include <cmath>

#include "umma_ptx.cuh"

namespace dfgpu {
namespace {

constexpr int kRows = 128;      // query rows of an item
constexpr int kKeys = 128;      // keys per tile
constexpr float kRescaleThreshold = 8.0f;  // log2 units

struct SdpaUmmaArgs {
    int32_t heads_q, seq_q, seq_kv;
    int32_t causal;
    int32_t order;            // of the work list: kAsStored, kHeavyWithLight, kHeaviestFirst or kLongestFirst (see ItemWalker)
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
    int32_t q_tiles;      // 128-row query tiles of a head, the last one perhaps partly past the end
    FastDivisor by_tiles, by_units, by_heads, by_batch_heads, by_group;   // query tiles and units of a head, query heads, all of them, query heads of a K/V head
    uint16_t* out;        // O, element strides by batch, head and position
    int64_t out_stride[3];
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

constexpr int kPolyEvery = 4;  // one pair of exponentials in kPolyEvery goes to the FMA pipe (0: none)
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

// ---- the kernel ------------------------------------------------------------------------------------
// A persistent CTA per SM walks a list of items, a query tile of 128 rows each, and its key tiles are one stream t = 0, 1, ... that runs on from
// item to item. (D is the head dimension.) Tensor memory: scores and probabilities of key tile t at 128 (t mod 3), O at 384 (two of them in
// turn for D = 64). P never goes through shared memory: each thread overwrites its own scores with 16-bit probabilities, two per column, and
// the second product takes its A operand from tensor memory. 24 warps:
//   warps 0-7, 8-15  softmax of the even and of the odd key tiles, two threads per query row (64 keys each; the two warps of a lane quarter trade row
//                    maxima through shared memory). The reference maximum of a row goes from tile to tile: each group passes it on as soon as it
//                    has seen its own tile's maximum, before its exponentials
//   warp 16          TMA: K and V in the order they are read: K0 K1 K2 V0 K3 V1 K4 ... through a ring of four slots
//   warp 17          issues the score products, up to three tiles ahead
//   warps 18-21      an item's end: its rows' sums of both groups, O out of tensor memory, normalised into a staging tile and off by TMA (left to the
//                    softmax warps it held up their next tile)
//   warp 22          issues the products with V
//   warp 23          TMA: Q, as soon as the last score product of the item before has read the old one (in the other loader's list it held up V)
// What bounds it, by clock stamps (a key tile of 128 x 128 of 2048 keys of 128 channels): 1024 clocks of products (GENERAL 1536), and a softmax
// of 2600 to 2900 (GENERAL 3300) on two groups. Three score tiles keep both busy: 1435 to 1600 clocks a tile (GENERAL 1830, near its products). With two
// query tiles of one SM, a score tile each, a tile's own chain of score product, softmax and second product set the pace (1835, 2200), and a
// causal or padded list was balanced to a pair of query tiles only. One warp issuing both kinds of product waited some 100 clocks before each, also
// for what had long arrived, with the tensor pipe idle: 2000 a tile. Code counts: 16 warps run it out of a small instruction cache, and an
// edge tile's masks compiled into the sixteens of every tile, or unrolled beside them, cost 3 to 7 %.
//   before (the better of that kernel and one that gave two SMs a pair) -> this, us a launch in a long row of them on changing operands (power limit):
//   4 x 16 (4) x 1000 x 128 padded causal 31.8 -> 28.7 (25 to 31 by the lengths), 32 heads of 2449 causal 115 -> 79, 21 x 8 x 796 causal 89 -> 66, 32 x 4096
//   causal 161 -> 152, 10 x 32 x 1895 x 64 padded 477 -> 434, 11 x 32 x 69 18.3 -> 10.4, 4 heads of 126 8.0 -> 6.5, 8 x 32 x 2048 causal 334 -> 329 (the first
//   twenty 284 -> 280, one by itself 313 -> 282). Short padded lists of 64 channels lost: 7 x 16 x 187 11.3 -> 11.8.
// GENERAL: what the kernel takes beyond whole tiles of packed bf16 rows of 128 (plain_tiles()): a batch's keys may end inside a key
// tile (padding masks, or a key length that is no multiple of 128), and probabilities are held to f32's accuracy: O += P V runs
// twice, on P rounded to the operands' type and on what that left over (16 or 22 bits in all), as O and Stats of these graphs are
// those of f32 probabilities (sdpa_rowwise_kernel's) to the rounding of O. PADDED: the batches have lengths of their own.
constexpr int kThreads = 24 * 32;
constexpr int kRingSlots = 4;
constexpr int kScoreTiles = 3;
constexpr int kMostListed = 1024;
template <int D>
struct SdpaSmem {
    static constexpr int kTile = kRows * D * 2;
    static constexpr int kQ = 0;
    static constexpr int kRing = kTile;
    static constexpr int kStage = kRing + kRingSlots * kTile;
    static constexpr int kMaxima = kStage + kTile;      // half-row maxima, bf16 (GENERAL: 24 bits as f32) [turn 2][group][quarter][half][lane]
    static constexpr int kReference = kMaxima + 4096;   // f32 [turn 2][group][half][quarter][lane]
    static constexpr int kSums = kReference + 4096;     // f32 {row sum, its reference, largest dot product} [group][half][row]
    static constexpr int kBarriers = kSums + 3 * 2048;
    static constexpr int kAccumulators = D == 64 ? 2 : 1;   // ... of D columns each: an item's is read out under the next one's products where there are two
    // sums_ready, sums_free, q_full, q_empty, o_full[2], o_empty[2], kv_full[S], kv_empty[S], s_full[3], p_full[3], pv_done[3], passed_on[group][half][quarter]
    static constexpr int kBarrierCount = 8 + 2 * kRingSlots + 3 * kScoreTiles + 16;
    static constexpr int kList = (kBarriers + kBarrierCount * 8 + 16 + 7) & ~7;   // kLongestFirst: (batch, query tile)s, 16 bits each
    static constexpr int kLengths = kList + 2 * kMostListed;           // ... and the batches' {keys, live query rows}
    static constexpr int kTotal = kLengths + 8 * kMostListed;
    static constexpr int kDynamic = kTotal + 1024;
    static_assert(kDynamic <= 227 * 1024, "the most a block may have");
};

// Key tiles of a query tile; none where no row of it has keys.
__device__ __forceinline__ int key_tiles(const SdpaUmmaArgs& args, int q_tile, int kv_len, int live_q) {
    if (q_tile * kRows >= live_q) return 0;
    const int kv_tiles = (kv_len + kKeys - 1) / kKeys;
    return args.causal ? min(kv_tiles, q_tile + 1) : kv_tiles;
}
struct QueryItem {
    int batch, head, kv_head;
    int q_tile, tiles;
    int kv_len;    // keys of this batch, at least one
    int live_q;    // query rows before this one have keys; the others store 0 and -inf
};
template <bool LENGTHS>
__device__ __forceinline__ void batch_lengths(const SdpaUmmaArgs& args, int batch, int& kv_len, int& live_q) {
    kv_len = args.seq_kv;
    live_q = args.seq_q;
    if (LENGTHS && args.len_q != nullptr) {
        const int len_kv = args.len_kv[batch * args.len_kv_stride], len_q = args.len_q[batch * args.len_q_stride];
        live_q = len_kv > 0 ? min(live_q, len_q) : 0;
        kv_len = max(1, min(kv_len, len_kv));
    }
}

// The work list of a CTA, the same in every warp role; query tiles without keys are left out of it (`every` takes them too).
//   kAsStored        head after head: CTA c takes items c, c + gridDim.x, ..., so that neighbours share a head's K and V in L2
//   kHeavyWithLight  causal: unit i of a head is the heavy tile T-1-i followed by the light tile i, so that every unit walks T+1 key tiles
//                    and equal numbers of units are equal work; neighbours share a head as above
//   kHeaviestFirst   causal: the query tiles of all heads by falling length, and every other round in reverse, so that the CTA with the
//                    longest tile of one round gets the shortest of the next
//   kLongestFirst    padded: the same by the key tiles that a batch's own lengths leave, in an order that each CTA works out for itself
enum { kAsStored = 0, kHeavyWithLight = 1, kHeaviestFirst = 2, kLongestFirst = 3 };
template <bool PADDED>
struct ItemWalker {
    int k = 0;
    const uint16_t* list = nullptr;
    const int2* lengths = nullptr;
    __device__ __forceinline__ bool next(const SdpaUmmaArgs& args, QueryItem& item, bool every = false) {
        const int places = static_cast<int>(gridDim.x), place = static_cast<int>(blockIdx.x), tiles = args.q_tiles;
        for (;;) {
            int bh;
            if (args.order == kHeavyWithLight) {
                const int unit = place + (k >> 1) * places, units = (tiles + 1) >> 1;
                if (unit >= units * args.batch_heads) return false;
                bh = static_cast<int>(fast_divide(unit, args.by_units));
                const int i = unit - bh * units;
                const bool light = (k & 1) != 0;
                ++k;
                if (light && 2 * i == tiles - 1) continue;   // the middle tile of an odd count stands alone
                item.q_tile = light ? i : tiles - 1 - i;
                item.batch = static_cast<int>(fast_divide(bh, args.by_heads));
                item.head = bh - item.batch * args.heads_q;
            } else {
                const int unit = k * places + (args.order != kAsStored && (k & 1) ? places - 1 - place : place);
                if (k * places >= tiles * args.batch_heads) return false;
                ++k;
                if (unit >= tiles * args.batch_heads) continue;   // (a reversed last round may have nothing for this place)
                if (PADDED && args.order == kLongestFirst) {
                    const int at = static_cast<int>(fast_divide(unit, args.by_heads)), entry = list[at];
                    item.batch = static_cast<int>(fast_divide(entry, args.by_tiles));
                    item.head = unit - at * args.heads_q;
                    item.q_tile = entry - item.batch * tiles;
                } else {
                    if (args.order == kAsStored) {
                        bh = static_cast<int>(fast_divide(unit, args.by_tiles));
                        item.q_tile = unit - bh * tiles;
                    } else {
                        const int at = static_cast<int>(fast_divide(unit, args.by_batch_heads));
                        bh = unit - at * args.batch_heads;
                        item.q_tile = tiles - 1 - at;
                    }
                    item.batch = static_cast<int>(fast_divide(bh, args.by_heads));
                    item.head = bh - item.batch * args.heads_q;
                }
            }
            item.kv_head = static_cast<int>(fast_divide(item.head, args.by_group));
            if (PADDED && args.order == kLongestFirst) {
                const int2 both = lengths[item.batch];
                item.kv_len = both.x;
                item.live_q = both.y;
            } else {
                batch_lengths<PADDED>(args, item.batch, item.kv_len, item.live_q);
            }
            item.tiles = key_tiles(args, item.q_tile, item.kv_len, item.live_q);
            if (PADDED && item.tiles == 0 && !every) continue;
            return true;
        }
    }
};
// The (batch, query tile)s, at most kMostListed, by falling number of key tiles, those of equal number as they are stored. A warp works out where an
// entry comes from the batches' lengths alone, a batch per lane.
__device__ __forceinline__ void longest_first(const SdpaUmmaArgs& args, uint16_t* list, int2* lengths) {
    const int batches = static_cast<int>(fast_divide(args.batch_heads, args.by_heads)), tiles = args.q_tiles, lane = threadIdx.x & 31;
    for (int b = static_cast<int>(threadIdx.x); b < batches; b += kThreads) batch_lengths<true>(args, b, lengths[b].x, lengths[b].y);
    __syncthreads();
    for (int own = static_cast<int>(threadIdx.x >> 5); own < batches * tiles; own += kThreads / 32) {
        const int batch = static_cast<int>(fast_divide(own, args.by_tiles)), q_tile = own - batch * tiles;
        const int weight = key_tiles(args, q_tile, lengths[batch].x, lengths[batch].y);
        int ahead = 0;
        for (int b = lane; b < batches; b += 32) {
            const int kv_tiles = (lengths[b].x + kKeys - 1) / kKeys, live = max(0, min(tiles, (lengths[b].y + kRows - 1) / kRows));
            // of this batch's query tiles, the ones with at least as many key tiles as `least`
            auto with = [&](int least) { return least <= 0 ? tiles : (kv_tiles < least ? 0 : (args.causal ? max(0, live - (least - 1)) : live)); };
            const int more = with(weight + 1), same = with(weight) - more;
            ahead += more;
            // (a batch's equal ones lie side by side: those without keys behind the live ones, under a causal mask the ones that see all keys)
            if (b < batch) ahead += same;
            else if (b == batch) ahead += q_tile - (weight == 0 ? live : (args.causal ? weight - 1 : 0));
        }
        ahead = __reduce_add_sync(0xffffffffu, ahead);
        if (lane == 0) list[ahead] = static_cast<uint16_t>(own);
    }
    __syncthreads();
}

// The key tiles of a CTA's work list, one after the other.
template <bool PADDED>
struct TileCursor {
    ItemWalker<PADDED> walker;
    QueryItem item;
    int j;        // key tile of the item
    uint32_t n;   // items before this one
    uint32_t t;   // key tiles before this one
    bool live;
    __device__ __forceinline__ void start(const SdpaUmmaArgs& args, const ItemWalker<PADDED>& from) {
        walker = from;
        n = t = 0;
        j = 0;
        live = walker.next(args, item);
    }
    __device__ __forceinline__ bool last() const { return j + 1 == item.tiles; }
    __device__ __forceinline__ void step(const SdpaUmmaArgs& args) {
        ++t;
        if (++j == item.tiles) {
            ++n;
            j = 0;
            live = walker.next(args, item);
        }
    }
};

template <int D, bool F16, bool GENERAL, bool PADDED>
__global__ void __launch_bounds__(kThreads, 1)
sdpa_umma_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v,
                      const __grid_constant__ CUtensorMap map_o, SdpaUmmaArgs args) {
    using Smem = SdpaSmem<D>;
    constexpr int kTileBytes = Smem::kTile;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t* generic_base = smem_raw + (smem_base - smem_u32(smem_raw));
    const uint32_t bar_base = smem_base + Smem::kBarriers;
    const uint32_t sums_ready = bar_base, sums_free = bar_base + 8, q_full = bar_base + 16, q_empty = bar_base + 24;
    constexpr uint32_t kAccumulators = Smem::kAccumulators;
    auto o_full = [&](uint32_t n) { return bar_base + 8u * (4 + n % kAccumulators); };
    auto o_empty = [&](uint32_t n) { return bar_base + 8u * (6 + n % kAccumulators); };
    auto o_parity = [](uint32_t n) { return (n / kAccumulators) & 1; };
    auto o_column = [](uint32_t n) { return 384 + n % kAccumulators * D; };
    auto kv_full = [&](uint32_t s) { return bar_base + 8u * (8 + s); };
    auto kv_empty = [&](uint32_t s) { return bar_base + 8u * (8 + kRingSlots + s); };
    auto s_full = [&](uint32_t b) { return bar_base + 8u * (8 + 2 * kRingSlots + b); };
    auto p_full = [&](uint32_t b) { return bar_base + 8u * (8 + 2 * kRingSlots + kScoreTiles + b); };
    auto pv_done = [&](uint32_t b) { return bar_base + 8u * (8 + 2 * kRingSlots + 2 * kScoreTiles + b); };
    auto passed_on = [&](int group, int half, int quarter) { return bar_base + 8u * (8 + 2 * kRingSlots + 3 * kScoreTiles + group * 8 + half * 4 + quarter); };
    const uint32_t tmem_slot = bar_base + 8u * Smem::kBarrierCount;
    volatile uint32_t* tmem_slot_ptr = reinterpret_cast<volatile uint32_t*>(generic_base + Smem::kBarriers + 8 * Smem::kBarrierCount);
    // ring place -> slot and the parity of its use
    auto slot_of = [](uint32_t place) { return place % kRingSlots; };
    auto parity_of = [](uint32_t place) { return (place / kRingSlots) & 1; };
    auto k_place = [](uint32_t t) { return t < 3 ? t : 2 * t - 2; };
    auto v_place = [](uint32_t t) { return 2 * t + 3; };

    const int warp = uniform_warp_index(), lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        prefetch_tensormap(&map_q);
        prefetch_tensormap(&map_k);
        prefetch_tensormap(&map_v);
        prefetch_tensormap(&map_o);
        mbar_init(sums_ready, 16);
        mbar_init(sums_free, 4);
        for (int n = 0; n < 2; ++n) {
            mbar_init(o_full(0) + 8u * n, 1);
            mbar_init(o_empty(0) + 8u * n, 4);
        }
        mbar_init(q_full, 1);
        mbar_init(q_empty, 1);
        for (int s = 0; s < kRingSlots; ++s) {
            mbar_init(kv_full(s), 1);
            mbar_init(kv_empty(s), 1);
        }
        for (int b = 0; b < kScoreTiles; ++b) {
            mbar_init(s_full(b), 1);
            mbar_init(p_full(b), 8);
            mbar_init(pv_done(b), 1);
        }
        for (int i = 0; i < 16; ++i) mbar_init(passed_on(0, 0, 0) + 8u * i, 1);
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
    ItemWalker<PADDED> beginning;
    beginning.list = reinterpret_cast<const uint16_t*>(generic_base + Smem::kList);
    beginning.lengths = reinterpret_cast<const int2*>(generic_base + Smem::kLengths);
    if (PADDED && args.order == kLongestFirst) longest_first(args, reinterpret_cast<uint16_t*>(generic_base + Smem::kList), reinterpret_cast<int2*>(generic_base + Smem::kLengths));
    chain_release();

    constexpr uint32_t kFormats = (1u << 4) | (F16 ? 0u : (1u << 7) | (1u << 10)) | (static_cast<uint32_t>(kRows >> 4) << 24);
    constexpr uint32_t kDescHi = smem_desc_hi(1024);
    if (warp == 16) {
        const bool leader = elect_one();
        TileCursor<PADDED> k, v;
        k.start(args, beginning);
        v.start(args, beginning);
        bool ok = true;
        auto put = [&](uint32_t place, const CUtensorMap* map, int row, int head, int batch) {
            const uint32_t slot = slot_of(place);
            if (ok) ok = mbar_wait_warp(kv_empty(slot), parity_of(place) ^ 1, 271);
            if (leader && ok) {
                mbar_expect_tx(kv_full(slot), kTileBytes);
#pragma unroll
                for (int h = 0; h < D / 64; ++h) tma_load_4d(smem_base + Smem::kRing + slot * kTileBytes + h * kHalfBytes, map, 64 * h, row, head, batch, kv_full(slot));
            }
            __syncwarp();
        };
        auto put_k = [&] {
            if (!k.live || !ok) return;
            put(k_place(k.t), &map_k, k.j * kKeys, k.item.kv_head, k.item.batch);
            k.step(args);
        };
        for (int i = 0; i < kScoreTiles; ++i) put_k();
        while (v.live && ok) {
            put(v_place(v.t), &map_v, v.j * kKeys, v.item.kv_head, v.item.batch);
            v.step(args);
            put_k();
        }
    } else if (warp == 23) {
        const bool leader = elect_one();
        ItemWalker<PADDED> walker = beginning;
        QueryItem item, following;
        bool ok = true, more = walker.next(args, item);
        for (uint32_t n = 0; more && ok; ++n) {
            ok = mbar_wait_warp(q_empty, (n & 1) ^ 1, 270);
            if (leader && ok) {
                mbar_expect_tx(q_full, kTileBytes);
#pragma unroll
                for (int h = 0; h < D / 64; ++h) tma_load_4d(smem_base + Smem::kQ + h * kHalfBytes, &map_q, 64 * h, item.q_tile * kRows, item.head, item.batch, q_full);
            }
            more = walker.next(args, following);
            if (leader && more) {   // (its copy has to wait for the buffer: from the L2 cache it takes half as long)
#pragma unroll
                for (int h = 0; h < D / 64; ++h) prefetch_box_4d(&map_q, 64 * h, following.q_tile * kRows, following.head, following.batch);
            }
            __syncwarp();
            item = following;
        }
    } else if (warp == 17) {
        const bool leader = elect_one();
        const uint32_t idesc_qk = kFormats | (static_cast<uint32_t>(kKeys >> 3) << 17) | args.negate_q;
        const uint32_t tmem_u = __shfl_sync(0xffffffffu, tmem_base, 0);
        TileCursor<PADDED> s;
        s.start(args, beginning);
        bool ok = true;
        while (s.live && ok) {
            const uint32_t b = s.t % kScoreTiles, place = k_place(s.t), slot = slot_of(place);
            if (s.j == 0) ok = mbar_wait_warp(q_full, s.n & 1, 272);
            if (ok) ok = mbar_wait_warp(kv_full(slot), parity_of(place), 273);
            if (ok) ok = mbar_wait_warp(pv_done(b), ((s.t / kScoreTiles) & 1) ^ 1, 286);   // (the probabilities that lay there have been multiplied)
            tc_fence_after();
            if (leader && ok) {
                const uint32_t q_lo = smem_desc_lo(smem_base + Smem::kQ, 16), k_lo = smem_desc_lo(smem_base + Smem::kRing + slot * kTileBytes, 16);
#pragma unroll
                for (int k = 0; k < D / 16; ++k) {
                    const uint32_t offset = ((k >> 2) * kHalfBytes + (k & 3) * 32) >> 4;   // in 16-byte units
                    umma_bf16(tmem_u + b * 128, desc_words(q_lo + offset, kDescHi), desc_words(k_lo + offset, kDescHi), idesc_qk, k != 0 ? 1u : 0u);
                }
                umma_commit(s_full(b));
                umma_commit(kv_empty(slot));
                if (s.last()) umma_commit(q_empty);
            }
            __syncwarp();
            s.step(args);
        }
    } else if (warp == 22) {
        const bool leader = elect_one();
        constexpr uint32_t idesc_pv = kFormats | (static_cast<uint32_t>(D >> 3) << 17) | (1u << 16);   // (V is read MN-major)
        const uint32_t tmem_u = __shfl_sync(0xffffffffu, tmem_base, 0);
        TileCursor<PADDED> p;
        p.start(args, beginning);
        bool ok = true;
        while (p.live && ok) {
            const uint32_t b = p.t % kScoreTiles, place = v_place(p.t), slot = slot_of(place), d_tmem = tmem_u + o_column(p.n);
            if (p.j == 0) ok = mbar_wait_warp(o_empty(p.n), o_parity(p.n) ^ 1, 274);
            // (V1's slot held K1, which this warp asks nothing of: the parity of V1's use could be that before K1's. The score product has read K1, and V0
            // and the later ones follow phases that this warp has waited for or that come first.)
            if (ok && p.t == 1) ok = mbar_wait_warp(s_full(b), 0, 277);
            if (ok) ok = mbar_wait_warp(kv_full(slot), parity_of(place), 275);
            if (ok) ok = mbar_wait_warp(p_full(b), (p.t / kScoreTiles) & 1, 276);
            tc_fence_after();
            if (leader && ok) {
                const uint32_t v_lo = smem_desc_lo(smem_base + Smem::kRing + slot * kTileBytes, kHalfBytes), p_tmem = tmem_u + b * 128;
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    const uint32_t p_at = p_tmem + (k >> 2) * 64 + (k & 3) * kProbabilityColumns<GENERAL>;
                    umma_bf16_a_tmem(d_tmem, p_at, desc_words(v_lo + ((k * 2048) >> 4), kDescHi), idesc_pv, (p.j | k) != 0 ? 1u : 0u);
                    if constexpr (GENERAL) umma_bf16_a_tmem(d_tmem, p_at + 8, desc_words(v_lo + ((k * 2048) >> 4), kDescHi), idesc_pv, 1u);
                }
                umma_commit(pv_done(b));
                umma_commit(kv_empty(slot));
                if (p.last()) umma_commit(o_full(p.n));
            }
            __syncwarp();
            p.step(args);
        }
    } else if (warp >= 18) {
        const int quarter = warp & 3, row = quarter * 32 + lane;
        const uint32_t lane_base = static_cast<uint32_t>(quarter * 32) << 16;
        const bool sender = warp == 18 && elect_one();
        const float* sums_of = reinterpret_cast<const float*>(generic_base + Smem::kSums) + row;   // + 512 * {sum, reference, largest} + (group * 2 + half) * 128
        auto meet = [] { asm volatile("bar.sync 9, 128;" ::: "memory"); };
        ItemWalker<PADDED> walker = beginning;
        QueryItem item;
        uint32_t n = 0, t0 = 0;
        bool ok = true;
        while (walker.next(args, item, true)) {   // (to the end also after a wait gave up: the warps meet at their barrier)
            if (PADDED && item.tiles == 0) {
                // No row of this query tile has keys: zeros and -inf, while these warps would wait for the next one's sums (a walk of its own at the end took 0.9 us,
                // with or without such tiles; by the softmax warps, in their shadow, its code cost every tile 3 to 8 %: 6 x 32 x 1748 x 64 122 us, 131).
                constexpr int kUnits = D / 8;   // of 16 bytes a row
                const int rows = min(kRows, args.seq_q - item.q_tile * kRows);
                const int64_t b64 = item.batch, h64 = item.head;
                for (int i = row; i < rows * kUnits; i += 128) {
                    const int64_t q64 = item.q_tile * kRows + i / kUnits;
                    *reinterpret_cast<uint4*>(args.out + b64 * args.out_stride[0] + h64 * args.out_stride[1] + q64 * args.out_stride[2] + (i % kUnits) * 8) = make_uint4(0, 0, 0, 0);
                }
                if (row < rows) {
                    const int64_t q64 = item.q_tile * kRows + row;
                    if (args.row_max != nullptr) args.row_max[b64 * args.max_stride[0] + h64 * args.max_stride[1] + q64 * args.max_stride[2]] = -INFINITY;
                    if (args.row_sum != nullptr) args.row_sum[b64 * args.sum_stride[0] + h64 * args.sum_stride[1] + q64 * args.sum_stride[2]] = 0.0f;
                    if (args.stats != nullptr) args.stats[b64 * args.stats_batch_stride + h64 * args.stats_head_stride + q64 * args.stats_row_stride] = -INFINITY;
                }
                continue;
            }
            const int q_index = item.q_tile * kRows + row;
            const int group = static_cast<int>((t0 + item.tiles - 1) & 1);   // of the item's last key tile, whose reference is the latest
            t0 += item.tiles;
            if (ok) ok = mbar_wait(sums_ready, n & 1, 283);
            float total = sums_of[group * 256] + sums_of[group * 256 + 128], row_raw_max = fmaxf(sums_of[group * 256 + 1024], sums_of[group * 256 + 128 + 1024]);
            const float m_ref = sums_of[512 + group * 256], other_ref = sums_of[512 + (group ^ 1) * 256];   // (both halves of a row know the same reference)
            if (other_ref != -INFINITY) {
                total += (sums_of[(group ^ 1) * 256] + sums_of[(group ^ 1) * 256 + 128]) * ex2_fast(other_ref - m_ref);
                row_raw_max = fmaxf(row_raw_max, fmaxf(sums_of[(group ^ 1) * 256 + 1024], sums_of[(group ^ 1) * 256 + 128 + 1024]));
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(sums_free);
            const bool live = !GENERAL || q_index < item.live_q;
            if (ok && q_index < args.seq_q) {
                const int64_t b64 = item.batch, h64 = item.head, q64 = q_index;
                if (args.row_max != nullptr)
                    args.row_max[b64 * args.max_stride[0] + h64 * args.max_stride[1] + q64 * args.max_stride[2]] = live ? row_raw_max * args.attn_scale : -INFINITY;
                if (args.row_sum != nullptr)
                    args.row_sum[b64 * args.sum_stride[0] + h64 * args.sum_stride[1] + q64 * args.sum_stride[2]] = live ? sum_against<GENERAL>(total, m_ref, row_raw_max * args.scale_log2) : 0.0f;
                if (args.stats != nullptr)
                    args.stats[b64 * args.stats_batch_stride + h64 * args.stats_head_stride + q64 * args.stats_row_stride] =
                        live ? natural_log_sum<GENERAL>(args, m_ref, total) : -INFINITY;
            }
            const float inverse = live ? inverse_of<GENERAL>(total) : 0.0f;
            if (sender) tma_store_wait_read<0>();   // (the staging tile's last copy)
            meet();
            if (ok) ok = mbar_wait(o_full(n), o_parity(n), 285);
            tc_fence_after();
            const uint32_t tmem_o = tmem_base + lane_base + o_column(n);
#pragma unroll 1
            for (int c = 0; c < D / 32; ++c) {
                uint32_t acc[32];
                tmem_load_32(tmem_o + c * 32, acc);
                tmem_load_wait();
                if (c == D / 32 - 1) {
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(o_empty(n));
                }
                uint8_t* o_row = generic_base + Smem::kStage + (c >> 1) * kHalfBytes + row * 128;
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    uint32_t w[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i)   // (selected, not multiplied: a dead row's accumulator may hold anything)
                        w[i] = live ? pack_pair<F16>(__uint_as_float(acc[u * 8 + 2 * i]) * inverse, __uint_as_float(acc[u * 8 + 2 * i + 1]) * inverse) : 0u;
                    *reinterpret_cast<uint4*>(o_row + ((((c & 1) * 4 + u) ^ (row & 7)) << 4)) = make_uint4(w[0], w[1], w[2], w[3]);
                }
            }
            fence_async_shared();
            meet();
            if (sender) {
                if (ok && g_device_status == 0) {
#pragma unroll
                    for (int h = 0; h < D / 64; ++h) tma_store_4d(&map_o, smem_base + Smem::kStage + h * kHalfBytes, 64 * h, item.q_tile * kRows, item.head, item.batch);
                }
                tma_store_commit();
            }
            ++n;
        }
        if (sender) tma_store_wait_all();
    } else {
        const int group = warp >> 3, half = (warp >> 2) & 1, quarter = warp & 3;
        const int row = quarter * 32 + lane;
        const uint32_t lane_base = static_cast<uint32_t>(quarter * 32) << 16;
        constexpr int kColumns = D / 2;   // of O per thread
        const float scale = args.scale_log2;
        const uint64_t scale2 = pack2(scale, scale);
        const int pair_barrier = 1 + group * 4 + quarter;   // the 64 threads of this group that share these 32 rows
        uint16_t* maxima = reinterpret_cast<uint16_t*>(generic_base + Smem::kMaxima) + (group * 4 + quarter) * 64 + lane;          // + turn * 512 + half * 32
        float* reference = reinterpret_cast<float*>(generic_base + Smem::kReference) + (half * 4 + quarter) * 32 + lane;           // + turn * 512 + group * 256
        float* sums_of = reinterpret_cast<float*>(generic_base + Smem::kSums) + row;   // + 512 * {sum, reference, largest} + (group * 2 + half) * 128
        uint32_t n = 0, t0 = 0;
        uint32_t mine_done = 0;   // key tiles this group has finished (parity of its maxima and references)
        bool ok = true;
        ItemWalker<PADDED> walker = beginning;
        QueryItem item;
        for (; walker.next(args, item); ++n) {   // (to the end also after a wait gave up: the warps of a row must meet at the same barriers)
            const int q_index = item.q_tile * kRows + row;
            const uint32_t tmem_o = tmem_base + lane_base + o_column(n) + half * kColumns;
            float m_ref = -INFINITY, l_sum = 0.0f, raw_max = -INFINITY;
            // The reference after key tile t, as the other group passed it on (tile t is the t / 2-th of its group).
            auto passed = [&](uint32_t t) {
                const uint32_t turn = t >> 1;
                if (ok) ok = mbar_wait(passed_on(group ^ 1, half, quarter), turn & 1, 278);
                return reference[(turn & 1) * 512 + (group ^ 1) * 256];
            };
            for (int j = static_cast<int>((t0 ^ group) & 1); j < item.tiles; j += 2, ++mine_done) {
                const uint32_t t = t0 + j, b = t % kScoreTiles;
                const uint32_t tmem_s = tmem_base + lane_base + b * 128 + half * 64;
                // (A wait tells a phase from its neighbours by parity alone, so the phase before must be over and the one behind it impossible. s_full(b):
                // S(t - 3) was over when the other group passed on tile t - 3, which this group took for tile t - 2, and S(t + 3) follows PV(t), which needs
                // this warp. passed_on: every phase is waited for, in order. pv_done(b): S(t) follows PV(t - 3), and PV(t + 1) follows PV(t).)
                if (ok) ok = mbar_wait(s_full(b), (t / kScoreTiles) & 1, 279);
                tc_fence_after();
                const int last_key = !GENERAL ? q_index : (args.causal ? min(q_index, item.kv_len - 1) : item.kv_len - 1);
                const int limit = last_key - j * kKeys - half * 64;
                const bool diagonal = (args.causal && j == item.q_tile) || (GENERAL && (j + 1) * kKeys > item.kv_len);
                // In a tile at the diagonal or at the batch's end: some rows of this warp have masked keys among these 64, and the last key that any of
                // them sees. Such tiles go sixteen keys at a time; the others are compiled without a branch between the sixteens.
                bool partly = false;
                int visible = 63;
                if (diagonal) {
                    partly = __reduce_min_sync(0xffffffffu, limit) < 63;
                    visible = min(63, __reduce_max_sync(0xffffffffu, limit));
                }
                auto masked = [&](uint32_t (&raw)[16], int c) {
                    if (partly) {
                        const int left = limit - c * 16;
#pragma unroll
                        for (int e = 0; e < 16; ++e)
                            if (e > left) raw[e] = 0xff800000u;  // -inf
                    }
                };
                // The tile's maximum first, then the reference, then the exponentials: nothing is formed twice. (The scores are read
                // twice, which costs next to nothing; 64 of them held in registers would spill.)
                float mine = -INFINITY;
                if (diagonal) {
#pragma unroll 1
                    for (int c = 0; c * 16 <= visible; ++c) {
                        uint32_t raw[16];
                        tmem_load_16(tmem_s + c * 16, raw);
                        tmem_load_wait_for(raw);
                        masked(raw, c);
                        mine = max_of_16(raw, mine);
                    }
                } else {
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
                        mine = max_of_16(raw[c + 1], max_of_16(raw[c], mine));
                    }
                }
                raw_max = fmaxf(raw_max, mine);
                // Trade the half-row maxima with the warp that owns the other 64 keys of these rows, as bf16 rounded towards +inf: any reference
                // not below the true maximum by more than the threshold serves, and both threads must arrive at the same value, so each uses
                // the rounded form of its own half too. (GENERAL: to 24 bits of the f32, since against a reference 2^-7 above a maximum of thousands all
                // probabilities would be zero; not the exact ones, with which Stats of 64 channels were 3.1e-8 from 64 bits for 2.4e-8. Two
                // buffers: the other warp may still be reading the last tile's when this one writes.)
                const uint32_t turn = mine_done & 1;
                float tile_max;
                if constexpr (GENERAL) {
                    float* exact = reinterpret_cast<float*>(generic_base + Smem::kMaxima) + (group * 4 + quarter) * 64 + lane;
                    const float up = __uint_as_float(round_up<24>(mine));
                    exact[turn * 512 + half * 32] = up;
                    asm volatile("bar.sync %0, 64;" ::"r"(pair_barrier) : "memory");
                    tile_max = fmaxf(up, exact[turn * 512 + (half ^ 1) * 32]) * scale;
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
                // (they go over columns whose scores have been read: 8 columns for every 16, or all 16)
                const uint64_t bias2 = pack2(bias_of<GENERAL>(m_ref), bias_of<GENERAL>(m_ref));
                if (diagonal) {
#pragma unroll 1
                    for (int c = 0; c < 4; ++c) {
                        const uint32_t at = tmem_s + c * kProbabilityColumns<GENERAL>;
                        if (c * 16 <= visible) {
                            uint32_t raw[16];
                            tmem_load_16(tmem_s + c * 16, raw);
                            tmem_load_wait_for(raw);
                            masked(raw, c);
                            put_probabilities<F16, GENERAL>(raw, scale2, bias2, sums, at);
                        } else {   // (no row of this warp sees these keys)
                            const uint32_t zeros[8] = {};
#pragma unroll
                            for (int column = 0; column < kProbabilityColumns<GENERAL>; column += 8) tmem_store_8(at + column, zeros);
                        }
                    }
                } else {
                    uint32_t raw[4][16];
                    tmem_load_16(tmem_s, raw[0]);
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        tmem_load_wait_for(raw[c]);
                        if (c < 3) tmem_load_16(tmem_s + (c + 1) * 16, raw[c + 1]);
                        put_probabilities<F16, GENERAL>(raw[c], scale2, bias2, sums, tmem_s + c * kProbabilityColumns<GENERAL>);
                    }
                }
                {
                    float lo, hi;
                    unpack2(add2(sums[0], sums[1]), lo, hi);
                    l_sum += lo + hi;
                }
                if (raise && j > 0) {
                    // O holds P V up to the tile before once that product is done; this tile's waits for these probabilities.
                    const float alpha = before == -INFINITY ? 0.0f : ex2_fast(before - m_new);
                    if (ok) ok = mbar_wait(pv_done((t - 1) % kScoreTiles), ((t - 1) / kScoreTiles) & 1, 280);
                    tc_fence_after();
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
                if (PADDED && (j + 1) * kKeys > item.kv_len && (D == 128 || half == 0)) {
                    // V rows past the batch's length are not this sequence's: cleared before the product
                    // (the slot held V(t - 2) before, which no wait above has asked for: while it is still on its way, its barrier is a phase further behind than
                    // the parity can tell. Once it has been multiplied, it has come. In the slot of V1 that was K1, which S(1) has read; V(t + 2) follows PV(t).)
                    const uint32_t place = v_place(t), v_slot = slot_of(place);
                    if (ok && t >= 2) ok = mbar_wait(pv_done((t - 2) % kScoreTiles), ((t - 2) / kScoreTiles) & 1, 284);
                    if (ok) ok = mbar_wait(kv_full(v_slot), parity_of(place), 281);
                    if (j * kKeys + row >= item.kv_len) {
                        uint8_t* v_row = generic_base + Smem::kRing + v_slot * kTileBytes + half * kHalfBytes + row * 128;
#pragma unroll
                        for (int u = 0; u < 8; ++u) *reinterpret_cast<uint4*>(v_row + ((u ^ (row & 7)) << 4)) = make_uint4(0, 0, 0, 0);   // (eight rows of a warp, eight different banks)
                    }
                    fence_async_shared();
                }
                tmem_store_wait();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(p_full(b));
            }
            // the item's end: what the warps that finish its rows need
            t0 += item.tiles;
            if (ok) ok = mbar_wait(sums_free, (n & 1) ^ 1, 282);   // (the last item's have been read)
            float* own = sums_of + (group * 2 + half) * 128;
            own[0] = l_sum;
            own[512] = m_ref;
            own[1024] = raw_max;
            __syncwarp();
            if (lane == 0) mbar_arrive(sums_ready);
        }
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 17) {
        tc_fence_after();
        tmem_dealloc(tmem_base, 512);
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
int launch_form(const CUtensorMap& map_q, const CUtensorMap& map_k, const CUtensorMap& map_v, const CUtensorMap& map_o, const SdpaUmmaArgs& args, unsigned grid, cudaStream_t stream) {
    cudaError_t error = cudaFuncSetAttribute(sdpa_umma_kernel<D, F16, GENERAL, PADDED>, cudaFuncAttributeMaxDynamicSharedMemorySize, SdpaSmem<D>::kDynamic);
    if (error != cudaSuccess) return fail(kExecutionFailed, "SDPA: cannot reserve %d bytes of shared memory: %s", SdpaSmem<D>::kDynamic, cudaGetErrorString(error));
    launch_chained(sdpa_umma_kernel<D, F16, GENERAL, PADDED>, dim3(grid), dim3(kThreads), SdpaSmem<D>::kDynamic, stream, map_q, map_k, map_v, map_o, args);
    return check_launch("SDPA (tcgen05)");
}
template <int D, bool F16>
int launch_general(const CUtensorMap& map_q, const CUtensorMap& map_k, const CUtensorMap& map_v, const CUtensorMap& map_o, const SdpaUmmaArgs& args, unsigned grid, cudaStream_t stream) {
    return args.len_q != nullptr ? launch_form<D, F16, true, true>(map_q, map_k, map_v, map_o, args, grid, stream)
                                 : launch_form<D, F16, true, false>(map_q, map_k, map_v, map_o, args, grid, stream);
}

bool packed_rows(const dfgpu_tensor& t) {
    return t.stride[3] == 1 && t.stride[2] == t.dim[3] && t.stride[1] == t.dim[2] * t.stride[2] && t.stride[0] == t.dim[1] * t.stride[1];
}
// Whole 128-row tiles of packed bf16 rows of 128, no padding, a causal mask on square scores only: P V on P rounded to bf16.
// (The kernel itself would take any number of query tiles and heads and a negative scale with Max and Sum_exp as well. Such graphs have had f32 probabilities
// ever since they ran on tensor cores, and in here they would get 16-bit ones.)
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
    return p.q.dim[0] * p.q.dim[1] * ((sq + 2 * kRows - 1) / (2 * kRows)) < (1ll << 30);   // (items, at most two for each of these, are counted in 31 bits)
}

int launch_sdpa_umma(const dfgpu_sdpa_params& p, void* const* tensors, cudaStream_t stream) {
    for (int i = 0; i < 4; ++i)
        if ((reinterpret_cast<uintptr_t>(tensors[i]) & 15u) != 0) return fail(kInvalidArgument, "SDPA: the tcgen05 kernel needs 16-byte aligned Q, K, V and O");
    CUtensorMap map_q, map_k, map_v, map_o;
    int status = sdpa_map(&map_q, p.q, tensors[0], kRows, "SDPA Q");
    if (!status) status = sdpa_map(&map_k, p.k, tensors[1], kKeys, "SDPA K");
    if (!status) status = sdpa_map(&map_v, p.v, tensors[2], kKeys, "SDPA V");
    if (!status) status = sdpa_map(&map_o, p.o, tensors[3], kRows, "SDPA O");
    if (status) return status;
    SdpaUmmaArgs args{};
    args.heads_q = static_cast<int>(p.q.dim[1]);
    args.seq_q = static_cast<int>(p.q.dim[2]);
    args.seq_kv = static_cast<int>(p.k.dim[2]);
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
    const int64_t heads = p.q.dim[0] * p.q.dim[1], kv_tiles = (p.k.dim[2] + kKeys - 1) / kKeys;
    args.q_tiles = static_cast<int>((p.q.dim[2] + kRows - 1) / kRows);
    args.out = static_cast<uint16_t*>(tensors[3]);
    for (int i = 0; i < 3; ++i) args.out_stride[i] = p.o.stride[i];
    args.by_tiles = make_fast_divisor(args.q_tiles);
    args.by_units = make_fast_divisor((args.q_tiles + 1) / 2);
    args.by_heads = make_fast_divisor(args.heads_q);
    args.by_batch_heads = make_fast_divisor(args.batch_heads);
    args.by_group = make_fast_divisor(args.heads_q / static_cast<int>(p.k.dim[1]));
    // The order of the list (see ItemWalker) where a CTA takes several items. Heaviest first, CTAs that run side by side read different heads' K and V, so only
    // where all of them stay in the L2 cache: 8 x 32 x 2048 causal, 268 MB of them, took 452 us that way in a short run, 274 as heavy and light tiles of
    // a head (29 x 4 x 1494, 88 MB: 54 and 64 the other way round). By length where lengths can differ by much: making the list costs each CTA 1 us, which
    // two or three key tiles a query tile do not give back unless there are many of them (31 x 8 x 25 16.8 us without, 13.6 with it; 27 x 4 x 167
    // 13.0 and 14.4; 16 x 32 x 303 x 64 35 and 32 the other way round), or the queries take more tiles than the keys: a head's last ones are likely behind their
    // batch's length then, and as stored, with an even number of them, half of the CTAs meet no others (16 x 16 x 512 on 128 keys x 64 21.2 without, 14.6 with it;
    // 7 x 16 x 256 on 128 11.1 and 10.3; 7 x 16 x 640 on 256, where few are, 16.3 and 16.7).
    const int64_t items = args.q_tiles * heads;
    const bool several = items > sm_count(), in_l2 = p.k.dim[0] * p.k.dim[1] * p.k.dim[2] * p.k.dim[3] * 4 <= (96 << 20);
    args.order = args.causal && several ? (in_l2 ? kHeaviestFirst : kHeavyWithLight) : kAsStored;
    const bool uneven = kv_tiles >= 4 || (kv_tiles >= 2 && items >= 4 * sm_count()) || (!args.causal && args.q_tiles > kv_tiles);
    if (p.padding_mask && several && in_l2 && uneven && p.q.dim[0] * args.q_tiles <= kMostListed) args.order = kLongestFirst;
    const int64_t units = args.order == kHeavyWithLight ? (args.q_tiles + 1) / 2 * heads : items;
    const unsigned grid = static_cast<unsigned>(std::min<int64_t>(units, sm_count()));
    if (plain_tiles(p)) return launch_form<128, false, false, false>(map_q, map_k, map_v, map_o, args, grid, stream);
    const bool f16 = p.q.dtype == DFGPU_F16;
    if (p.q.dim[3] == 64) return f16 ? launch_general<64, true>(map_q, map_k, map_v, map_o, args, grid, stream) : launch_general<64, false>(map_q, map_k, map_v, map_o, args, grid, stream);
    return f16 ? launch_general<128, true>(map_q, map_k, map_v, map_o, args, grid, stream) : launch_general<128, false>(map_q, map_k, map_v, map_o, args, grid, stream);
}

int sdpa_umma_device_status(int* status) { return read_and_clear_device_status(status); }

}  // namespace dfgpu
