// MATMUL on CUDA cores: batched, broadcast over leading axes, arbitrary strides,
// f32 accumulation. With block scales attached, A and/or B are E4M3 codes that are
// decoded and multiplied by their E8M0 block scale while the tile is staged, which
// absorbs the BLOCK_SCALE_DEQUANTIZE nodes in front of the MATMUL. The tcgen05
// kernels in umma_matmul.cu and umma_conv_f32.cu take over wherever they can read the operands.
#include <cooperative_groups.h>

#include <algorithm>

#include "common.cuh"
#include "umma.cuh"

namespace dfgpu {
namespace {

struct MatmulArgs {
    View a, b, c;
    View a_scale, b_scale;
    const uint8_t* a_scale_data;
    const uint8_t* b_scale_data;
    int64_t a_block[2], b_block[2];
    View extra[2];
    const void* extra_data[2];
    Epilogue epilogue;
    int rank;
    int64_t m, n, k;
};

__device__ __forceinline__ void batch_offsets(const MatmulArgs& g, int64_t batch, int64_t& ao, int64_t& bo, int64_t& co,
                                              int64_t& aso, int64_t& bso, int64_t* batch_index) {
    ao = bo = co = aso = bso = 0;
    for (int i = g.rank - 3; i >= 0; --i) {
        int64_t position = batch % g.c.dim[i];
        batch /= g.c.dim[i];
        batch_index[i] = position;
        ao += (g.a.dim[i] == 1 ? 0 : position) * g.a.stride[i];
        bo += (g.b.dim[i] == 1 ? 0 : position) * g.b.stride[i];
        co += position * g.c.stride[i];
        if (g.a_scale.rank) aso += (g.a_scale.dim[i] == 1 ? 0 : position) * g.a_scale.stride[i];
        if (g.b_scale.rank) bso += (g.b_scale.dim[i] == 1 ? 0 : position) * g.b_scale.stride[i];
    }
}

__device__ __forceinline__ float fused_steps(const MatmulArgs& g, float value, int64_t m, int64_t n, const int64_t* batch_index) {
    const int r = g.rank;
    for (int step = 0; step < g.epilogue.count; ++step) {
        if (g.epilogue.op[step] == DFGPU_EPI_ADD) {
            const View& t = g.extra[g.epilogue.operand[step]];
            int shift = r - t.rank;
            int64_t offset = 0;
            for (int axis = 0; axis < t.rank; ++axis) {
                int out_axis = axis + shift;
                int64_t position = out_axis == r - 1 ? n : (out_axis == r - 2 ? m : batch_index[out_axis]);
                offset += (t.dim[axis] == 1 ? 0 : position) * t.stride[axis];
            }
            value = __fadd_rn(value, load_as_f32(g.extra_data[g.epilogue.operand[step]], t.dtype, offset));
        } else {
            value = relu_forward(value, g.epilogue.lower[step], g.epilogue.upper[step], g.epilogue.slope[step]);
        }
    }
    return value;
}

__global__ void __launch_bounds__(256)
matmul_ffma_kernel(const void* __restrict__ a, const void* __restrict__ b, void* __restrict__ c, MatmulArgs g, const int* __restrict__ run_if_any,
                   int flag_count) {
    chain_begin();
    a = after_chain(a);
    b = after_chain(b);
    run_if_any = after_chain(run_if_any);
    constexpr int BM = 64, BN = 64, BK = 16, TM = 4, TN = 4;
    __shared__ float as[BK][BM + 4];
    __shared__ float bs[BK][BN + 4];
    const int tid = threadIdx.x;
    if (run_if_any) {
        // second pass behind the split-operand tensor-core form: it only has work when one of the flags is set
        int any = 0;
        for (int i = tid; i < flag_count; i += 256) any |= run_if_any[i];
        if (!__syncthreads_or(any)) return;
    }
    // (one tile per CTA, except behind the tensor-core form, whose check costs less with fewer CTAs)
    for (int64_t m0 = static_cast<int64_t>(blockIdx.x) * BM; m0 < g.m; m0 += static_cast<int64_t>(gridDim.x) * BM)
    for (int64_t n0 = static_cast<int64_t>(blockIdx.y) * BN; n0 < g.n; n0 += static_cast<int64_t>(gridDim.y) * BN) {
    int64_t batch_index[DFGPU_MAX_RANK];
    int64_t ao, bo, co, aso, bso;
    batch_offsets(g, blockIdx.z, ao, bo, co, aso, bso, batch_index);
    const int r = g.rank;
    // A is read k-fastest when its k stride is 1, else m-fastest; same idea for B.
    const bool a_k_fast = g.a.stride[r - 1] == 1;
    const bool b_n_fast = g.b.stride[r - 1] == 1;
    const int ty = tid / 16, tx = tid % 16;
    float acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = 0.0f;

    for (int64_t k0 = 0; k0 < g.k; k0 += BK) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            int e = tid + i * 256;
            int mm = a_k_fast ? e / BK : e % BM;
            int kk = a_k_fast ? e % BK : e / BM;
            int64_t m = m0 + mm, k = k0 + kk;
            float value = 0.0f;
            if (m < g.m && k < g.k) {
                value = load_as_f32(a, g.a.dtype, ao + m * g.a.stride[r - 2] + k * g.a.stride[r - 1]);
                if (g.a_scale.rank)
                    value = __fmul_rn(value, decode_e8m0(g.a_scale_data[aso + (m / g.a_block[0]) * g.a_scale.stride[r - 2] +
                                                                           (k / g.a_block[1]) * g.a_scale.stride[r - 1]]));
            }
            as[kk][mm] = value;
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            int e = tid + i * 256;
            int nn = b_n_fast ? e % BN : e / BK;
            int kk = b_n_fast ? e / BN : e % BK;
            int64_t n = n0 + nn, k = k0 + kk;
            float value = 0.0f;
            if (n < g.n && k < g.k) {
                value = load_as_f32(b, g.b.dtype, bo + k * g.b.stride[r - 2] + n * g.b.stride[r - 1]);
                if (g.b_scale.rank)
                    value = __fmul_rn(value, decode_e8m0(g.b_scale_data[bso + (k / g.b_block[0]) * g.b_scale.stride[r - 2] +
                                                                           (n / g.b_block[1]) * g.b_scale.stride[r - 1]]));
            }
            bs[kk][nn] = value;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < BK; ++kk) {
            float av[TM], bv[TN];
#pragma unroll
            for (int i = 0; i < TM; ++i) av[i] = as[kk][ty * TM + i];
#pragma unroll
            for (int j = 0; j < TN; ++j) bv[j] = bs[kk][tx * TN + j];
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
        }
        __syncthreads();
    }

#pragma unroll
    for (int i = 0; i < TM; ++i) {
        int64_t m = m0 + ty * TM + i;
        if (m >= g.m) continue;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            int64_t n = n0 + tx * TN + j;
            if (n >= g.n) continue;
            const float value = fused_steps(g, acc[i][j], m, n, batch_index);
            store_from_f32(c, g.c.dtype, co + m * g.c.stride[r - 2] + n * g.c.stride[r - 1], value);
        }
    }
    }
}

// ---- few rows of f32: C[M, N] with M <= kFewRows ---------------------------------------------------------------
// Bound by reading B once, so nothing but enough loads in flight matters: a CTA takes 32 columns and a share of K (a cluster
// shares out the K of its columns), 128 of K at a time, each thread four float4 of B, the next four already on their way. A
// comes through shared memory. 1 x 4096 x 4096: 17 us, 16 rows 38, the tensor-core form 59 whatever the rows (it splits B into
// pieces either way); at 32 rows the products bound this one (1688 columns, 4232 deep: 39 us against 27).
//   K contiguous in B:  warp w the columns 4 w .. 4 w + 3, lane l the depths 4 l .. 4 l + 3 of the 128
//   N contiguous in B:  8 lanes the 32 columns, 4 each, of one row; the 32 groups of 8 lanes four rows each
// Either way a thread holds a 4 x 4 block of B. Sums run in f32 over 1/32 of the CTA's depth per thread, then as a tree.
constexpr int kFewColumns = 32, kFewDepth = 128;
constexpr int kFewRows = 16;

template <int ROWS, bool B_K_MAJOR>
__global__ void __launch_bounds__(256)
matmul_few_rows_kernel(const float* __restrict__ a, const float* __restrict__ b, void* __restrict__ c, const __grid_constant__ MatmulArgs g, int64_t a_ld, int64_t a_step,
                       int64_t b_ld, int chunks_per_cta) {
    namespace cg = cooperative_groups;
    constexpr int kSums = ROWS * 4;
    __shared__ __align__(16) float as[2][ROWS][kFewDepth];
    __shared__ __align__(16) float partial[8][ROWS][kFewColumns];   // by warp; then [0] holds the CTA's sums
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    cg::cluster_group cluster = cg::this_cluster();
    const int rank = static_cast<int>(cluster.block_rank()), ranks = static_cast<int>(cluster.num_blocks());
    const int K = static_cast<int>(g.k), N = static_cast<int>(g.n), n0 = blockIdx.y * kFewColumns, m0 = blockIdx.z * ROWS;
    const int rows = min(ROWS, static_cast<int>(g.m) - m0);
    const int first_chunk = rank * chunks_per_cta, chunks = max(0, min((K + kFewDepth - 1) / kFewDepth - first_chunk, chunks_per_cta));
    const int column = n0 + (B_K_MAJOR ? warp * 4 : (lane & 7) * 4), depth = B_K_MAJOR ? lane * 4 : (warp * 4 + (lane >> 3)) * 4;
    const float4 zero = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    chain_wait();
    chain_release();
    a = after_chain(a);
    b = after_chain(b);
    auto fetch_b = [&](int chunk, float4 (&v)[4]) {
        const int k = (first_chunk + chunk) * kFewDepth + depth;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const bool live = B_K_MAJOR ? k < K && column + j < N : k + j < K && column < N;
            v[j] = live ? __ldg(reinterpret_cast<const float4*>(B_K_MAJOR ? b + (column + j) * b_ld + k : b + (k + j) * b_ld + column)) : zero;
        }
    };
    constexpr int kPerThread = (ROWS * kFewDepth + 255) / 256;
    auto fetch_a = [&](int chunk, float (&v)[kPerThread]) {
#pragma unroll
        for (int j = 0; j < kPerThread; ++j) {
            const int at = tid + j * 256, row = at / kFewDepth, k = (first_chunk + chunk) * kFewDepth + at % kFewDepth;
            v[j] = row < rows && k < K ? __ldg(a + (m0 + row) * a_ld + k * a_step) : 0.0f;
        }
    };
    float sum[kSums];   // [row][column]
#pragma unroll
    for (int i = 0; i < kSums; ++i) sum[i] = 0.0f;
    float4 bv[4], bn[4];
    float av[kPerThread];
    if (chunks > 0) {
        fetch_b(0, bv);
        fetch_a(0, av);
    }
    for (int chunk = 0; chunk < chunks; ++chunk) {
        float(&tile)[ROWS][kFewDepth] = as[chunk & 1];
#pragma unroll
        for (int j = 0; j < kPerThread; ++j)
            if (ROWS * kFewDepth >= 256 || tid < ROWS * kFewDepth) (&tile[0][0])[tid + j * 256] = av[j];
        if (chunk + 1 < chunks) {
            fetch_b(chunk + 1, bn);
            fetch_a(chunk + 1, av);
        }
        __syncthreads();   // (the tile written two chunks on was read before this one's barrier)
#pragma unroll
        for (int row = 0; row < ROWS; ++row) {
            const float4 x = *reinterpret_cast<const float4*>(&tile[row][depth]);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                if constexpr (B_K_MAJOR) {
                    sum[row * 4 + j] = fmaf(x.w, bv[j].w, fmaf(x.z, bv[j].z, fmaf(x.y, bv[j].y, fmaf(x.x, bv[j].x, sum[row * 4 + j]))));
                } else {
                    const float xj = j == 0 ? x.x : (j == 1 ? x.y : (j == 2 ? x.z : x.w));
                    sum[row * 4] = fmaf(xj, bv[j].x, sum[row * 4]);
                    sum[row * 4 + 1] = fmaf(xj, bv[j].y, sum[row * 4 + 1]);
                    sum[row * 4 + 2] = fmaf(xj, bv[j].z, sum[row * 4 + 2]);
                    sum[row * 4 + 3] = fmaf(xj, bv[j].w, sum[row * 4 + 3]);
                }
            }
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) bv[j] = bn[j];
    }
    // The lanes that share columns (all 32, or those 8 and 16 apart): each level halves what a lane still holds, a lane keeping
    // the upper half where its bit of the index is set, until one value is left, which the remaining levels add up.
    int held = kSums, first = 0;   // (both known at compile time once unrolled; `first` is the lane's)
#pragma unroll
    for (int bit = B_K_MAJOR ? 1 : 8; bit < 32; bit *= 2) {
        if (held > 1) {
            held /= 2;
            const bool upper = (lane & bit) != 0;
#pragma unroll
            for (int i = 0; i < kSums / 2; ++i) {
                if (i >= held) break;
                const float give = upper ? sum[i] : sum[i + held], keep = upper ? sum[i + held] : sum[i];
                sum[i] = keep + __shfl_xor_sync(0xffffffffu, give, bit);
            }
            if (upper) first += held;
        } else {
            sum[0] += __shfl_xor_sync(0xffffffffu, sum[0], bit);
        }
    }
#pragma unroll
    for (int i = 0; i < kSums; ++i) {
        if (i >= held) break;
        const int at = first + i, row = at >> 2, col = (B_K_MAJOR ? warp * 4 : (lane & 7) * 4) + (at & 3);
        partial[B_K_MAJOR ? 0 : warp][row][col] = sum[i];
    }
    if constexpr (!B_K_MAJOR) {
        __syncthreads();
        for (int at = tid; at < ROWS * kFewColumns; at += 256) {
            float total = (&partial[0][0][0])[at];
#pragma unroll
            for (int w = 1; w < 8; ++w) total += (&partial[w][0][0])[at];
            (&partial[0][0][0])[at] = total;   // (every element is read and written by one thread)
        }
    }
    cluster.sync();
    const int64_t no_batch[DFGPU_MAX_RANK] = {};
    const int r = g.rank;
    bool rare = false;
    for (int at = rank * 256 + tid; at < rows * kFewColumns; at += ranks * 256) {
        const int64_t m = m0 + at / kFewColumns, n = n0 + at % kFewColumns;
        if (n >= N) continue;
        float value = 0.0f;
        for (int z = 0; z < ranks; ++z) value += cluster.map_shared_rank(&partial[0][0][0], z)[at];
        rare = rare || __float_as_uint(value) == kRareSum;
        store_from_f32(c, g.c.dtype, m * g.c.stride[r - 2] + n * g.c.stride[r - 1], fused_steps(g, value, m, n, no_batch));
    }
    // No CTA leaves while another still reads its sums. (Nothing is published with it, and a release would wait for the stores of C.)
    __syncwarp();
    cluster_arrive_behind_loads(rare);
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

struct FewRows {
    bool b_k_major;
    int64_t a_ld, a_step, b_ld;
};
bool few_rows_form(const dfgpu_matmul_params& p, FewRows& form) {
    if (p.a.dtype != DFGPU_F32 || p.b.dtype != DFGPU_F32 || p.a_scale.rank || p.b_scale.rank) return false;
    const int rank = p.c.rank;
    if (rank < 2 || p.a.rank != rank || p.b.rank != rank) return false;
    for (int i = 0; i < rank - 2; ++i)
        if (p.c.dim[i] != 1 || p.a.dim[i] != 1 || p.b.dim[i] != 1) return false;
    const int64_t M = p.c.dim[rank - 2], N = p.c.dim[rank - 1], K = p.a.dim[rank - 1];
    if (M < 1 || M > kFewRows || N < 1 || K < 1 || N > 65535ll * kFewColumns || K >= (1ll << 30)) return false;   // (grid extents; 32-bit depths)
    form.a_ld = p.a.stride[rank - 2];
    form.a_step = p.a.stride[rank - 1];
    // float4 loads of B: contiguous rows of whole float4s on 16-byte boundaries
    form.b_k_major = p.b.stride[rank - 2] == 1 && K % 4 == 0 && p.b.stride[rank - 1] % 4 == 0;
    form.b_ld = p.b.stride[form.b_k_major ? rank - 1 : rank - 2];
    return form.b_k_major || (p.b.stride[rank - 1] == 1 && N % 4 == 0 && form.b_ld % 4 == 0);
}

template <int ROWS>
cudaError_t launch_few_rows(const FewRows& form, const MatmulArgs& g, void* const* tensors, cudaStream_t stream) {
    const int tiles = static_cast<int>((g.n + kFewColumns - 1) / kFewColumns), row_tiles = static_cast<int>((g.m + ROWS - 1) / ROWS);
    const int chunks = static_cast<int>((g.k + kFewDepth - 1) / kFewDepth);
    // K is shared out until every SM has two CTAs; a CTA without a chunk only adds zeros
    const int wanted = std::min(std::min(8, chunks), std::max(1, (2 * 148 + tiles * row_tiles - 1) / (tiles * row_tiles)));
    const int per_cta = (chunks + wanted - 1) / wanted, ranks = (chunks + per_cta - 1) / per_cta;
    auto kernel = form.b_k_major ? matmul_few_rows_kernel<ROWS, true> : matmul_few_rows_kernel<ROWS, false>;
    return launch_chained_cluster(kernel, dim3(static_cast<unsigned>(ranks), static_cast<unsigned>(tiles), static_cast<unsigned>(row_tiles)), dim3(256), static_cast<unsigned>(ranks),
                                  0, stream, static_cast<const float*>(tensors[0]), static_cast<const float*>(tensors[1]), tensors[2], g, form.a_ld, form.a_step, form.b_ld, per_cta);
}
int launch_few_rows(const FewRows& form, const MatmulArgs& g, void* const* tensors, cudaStream_t stream) {
    cudaError_t error;
    if (g.m <= 1) error = launch_few_rows<1>(form, g, tensors, stream);
    else if (g.m <= 2) error = launch_few_rows<2>(form, g, tensors, stream);
    else if (g.m <= 4) error = launch_few_rows<4>(form, g, tensors, stream);
    else if (g.m <= 8) error = launch_few_rows<8>(form, g, tensors, stream);
    else error = launch_few_rows<16>(form, g, tensors, stream);
    if (error != cudaSuccess) return fail(kExecutionFailed, "MATMUL: cluster launch failed: %s", cudaGetErrorString(error));
    return check_launch("MATMUL");
}

int build_args(const dfgpu_matmul_params& p, void* const* tensors, MatmulArgs& g) {
    if (!valid_tensor(p.a) || !valid_tensor(p.b) || !valid_tensor(p.c))
        return fail(kInvalidShape, "MATMUL: tensor rank or extent out of range");
    int rank = p.c.rank;
    if (rank < 2 || p.a.rank != rank || p.b.rank != rank) return fail(kInvalidShape, "MATMUL: A, B and C must have equal rank >= 2");
    int64_t m = p.c.dim[rank - 2], n = p.c.dim[rank - 1], k = p.a.dim[rank - 1];
    if (p.a.dim[rank - 2] != m || p.b.dim[rank - 1] != n || p.b.dim[rank - 2] != k)
        return fail(kInvalidShape, "MATMUL: M/N/K extents are inconsistent");
    for (int i = 0; i < rank - 2; ++i) {
        if ((p.a.dim[i] != 1 && p.a.dim[i] != p.c.dim[i]) || (p.b.dim[i] != 1 && p.b.dim[i] != p.c.dim[i]))
            return fail(kInvalidShape, "MATMUL: batch axes do not broadcast");
    }
    auto float_type = [](int t) { return t == DFGPU_F32 || t == DFGPU_F16 || t == DFGPU_BF16; };
    const dfgpu_tensor* operands[2] = {&p.a, &p.b};
    const dfgpu_tensor* scales[2] = {&p.a_scale, &p.b_scale};
    const int64_t* blocks[2] = {p.a_block, p.b_block};
    for (int which = 0; which < 2; ++which) {
        const dfgpu_tensor& t = *operands[which];
        const dfgpu_tensor& s = *scales[which];
        if (s.rank == 0) {
            if (!float_type(t.dtype)) return fail(kUnsupported, "MATMUL: operand must be FLOAT, HALF or BFLOAT16 unless block scales are attached");
            continue;
        }
        if (t.dtype != DFGPU_E4M3 || s.dtype != DFGPU_E8M0 || s.reorder != DFGPU_REORDER_NONE)
            return fail(kUnsupported, "MATMUL: fused dequantize takes FP8_E4M3 codes with unreordered FP8_E8M0 scales");
        if (s.rank != rank || blocks[which][0] <= 0 || blocks[which][1] <= 0)
            return fail(kInvalidShape, "MATMUL: block scale descriptor is inconsistent");
        for (int axis = rank - 2; axis < rank; ++axis) {
            int64_t block = blocks[which][axis - (rank - 2)];
            if (s.dim[axis] < (t.dim[axis] + block - 1) / block) return fail(kInvalidShape, "MATMUL: block scale tensor smaller than the block grid");
        }
    }
    if (!float_type(p.c.dtype)) return fail(kUnsupported, "MATMUL: C must be FLOAT, HALF or BFLOAT16");
    int status = validate_epilogue(p.epilogue_count, p.epilogue, p.extra, tensors ? tensors + 5 : nullptr, p.c, "MATMUL");
    if (status) return status;
    g.a = make_view(p.a);
    g.b = make_view(p.b);
    g.c = make_view(p.c);
    g.a_scale = make_view(p.a_scale);
    g.b_scale = make_view(p.b_scale);
    g.a_scale.rank = p.a_scale.rank;
    g.b_scale.rank = p.b_scale.rank;
    g.a_scale_data = tensors ? static_cast<const uint8_t*>(tensors[3]) : nullptr;
    g.b_scale_data = tensors ? static_cast<const uint8_t*>(tensors[4]) : nullptr;
    for (int i = 0; i < 2; ++i) {
        g.a_block[i] = p.a_block[i] > 0 ? p.a_block[i] : 1;
        g.b_block[i] = p.b_block[i] > 0 ? p.b_block[i] : 1;
        g.extra[i] = make_view(p.extra[i]);
        g.extra_data[i] = tensors ? tensors[5 + i] : nullptr;
    }
    g.epilogue = make_epilogue(p.epilogue_count, p.epilogue);
    g.rank = rank;
    g.m = m;
    g.n = n;
    g.k = k;
    return kOk;
}

// ---- f32 matmul on the bf16 tensor cores (split_f32.cu) ----------------------------------------------------
struct SplitMatmul {
    PieceOperand a, b;         // (pointers and `vector` filled in at launch)
    PieceMatmul product;
    int64_t b_offset, flags_offset, scratch_bytes;
    int flag_count;
};

// Takes unbatched f32 A [M, K] with K contiguous, f32 B with N or K contiguous and a row-major C.
bool f32_split_matmul(const dfgpu_matmul_params& p, SplitMatmul& form) {
    if (p.a.dtype != DFGPU_F32 || p.b.dtype != DFGPU_F32 || p.c.dtype != DFGPU_F32 || p.a_scale.rank || p.b_scale.rank) return false;
    const int rank = p.c.rank;
    if (rank < 2 || p.a.rank != rank || p.b.rank != rank) return false;
    for (int i = 0; i < rank - 2; ++i)
        if (p.c.dim[i] != 1 || p.a.dim[i] != 1 || p.b.dim[i] != 1) return false;
    const int64_t M = p.c.dim[rank - 2], N = p.c.dim[rank - 1], K = p.a.dim[rank - 1];
    if (M < 1 || N < 1 || K < 1 || M * K >= (1ll << 29) || K * N >= (1ll << 29) || std::max(M, N) >= (1ll << 28)) return false;
    if (p.a.stride[rank - 1] != 1 || p.a.stride[rank - 2] < K) return false;
    const bool b_n_major = p.b.stride[rank - 1] == 1 && p.b.stride[rank - 2] >= N;
    const bool b_k_major = !b_n_major && p.b.stride[rank - 2] == 1 && p.b.stride[rank - 1] >= K;
    if ((!b_n_major && !b_k_major) || !matmul_pieces_supported(p)) return false;
    auto operand = [](int64_t rows, int64_t length, int64_t source_ld) {
        PieceOperand o{};
        o.row_groups = static_cast<int32_t>((length + 3) / 4);
        o.groups = static_cast<int32_t>(rows * o.row_groups);
        o.row_length = static_cast<int32_t>(length);
        o.by_row = make_fast_divisor(static_cast<uint32_t>(o.row_groups));
        o.source_ld = source_ld;
        o.out_ld = (length + 7) / 8 * 8;
        o.piece_stride = rows * o.out_ld;
        return o;
    };
    form.a = operand(M, K, p.a.stride[rank - 2]);
    form.b = b_n_major ? operand(K, N, p.b.stride[rank - 2]) : operand(N, K, p.b.stride[rank - 1]);
    if (form.a.piece_stride >= (1ll << 29) || form.b.piece_stride >= (1ll << 29)) return false;
    form.product = PieceMatmul{nullptr, nullptr, form.a.out_ld, form.b.out_ld, b_n_major};
    auto round_up = [](int64_t v) { return (v + 255) / 256 * 256; };
    form.flag_count = piece_flag_count(form.a, form.b);
    form.b_offset = round_up(form.a.piece_stride * 6);
    form.flags_offset = form.b_offset + round_up(form.b.piece_stride * 6);
    form.scratch_bytes = form.flags_offset + round_up(static_cast<int64_t>(form.flag_count) * 4);
    return true;
}

int choose_kernel(const dfgpu_matmul_params& p, int& kernel) {
    int automatic = DFGPU_MATMUL_FFMA;
    SplitMatmul split;
    const bool split_ok = f32_split_matmul(p, split);
    if (matmul_umma_supported(p, DFGPU_MATMUL_UMMA_MXF8)) automatic = DFGPU_MATMUL_UMMA_MXF8;
    else if (matmul_umma_supported(p, DFGPU_MATMUL_UMMA_BF16)) automatic = DFGPU_MATMUL_UMMA_BF16;
    else if (FewRows few; few_rows_form(p, few)) automatic = DFGPU_MATMUL_FFMA;
    else {
        const int64_t macs = p.c.dim[p.c.rank - 2] * p.c.dim[p.c.rank - 1] * p.a.dim[p.a.rank - 1];
        if (split_ok && macs >= kSplitFormMinMacs) automatic = DFGPU_MATMUL_UMMA_F32X3;  // (three launches: big products only)
        // (one launch beats three where the output tiles fit one wave, 17 us against 22 at 512 x 2048 x 512, 34 against 24 at
        // 2048 x 512 x 1024, or all columns fit one tile, 64 against 118 at 30000 x 1024 x 64)
        const int64_t row_tiles = (p.c.dim[p.c.rank - 2] + 127) / 128, column_tiles = (p.c.dim[p.c.rank - 1] + 63) / 64;
        const bool one_launch_pays = automatic != DFGPU_MATMUL_UMMA_F32X3 || row_tiles * column_tiles <= 148 || column_tiles == 1;
        if (one_launch_pays && p.a.dim[p.a.rank - 1] >= kClusterFormMinDepth && matmul_f32_cluster_supported(p)) automatic = DFGPU_MATMUL_UMMA_F32X3_CLUSTER;
    }
    kernel = p.kernel == DFGPU_MATMUL_AUTO ? automatic : p.kernel;
    if (kernel < DFGPU_MATMUL_FFMA || kernel > DFGPU_MATMUL_UMMA_F32X3_CLUSTER) return fail(kInvalidArgument, "MATMUL: unknown kernel id %d", kernel);
    if (kernel == DFGPU_MATMUL_UMMA_F32X3_CLUSTER) {
        if (!matmul_f32_cluster_supported(p))
            return fail(kUnsupported, "MATMUL: the one-launch tcgen05 form needs FLOAT, HALF or BFLOAT16 A, B and C and at most one batch axis");
        return kOk;
    }
    if (kernel == DFGPU_MATMUL_UMMA_F32X3) {
        if (!split_ok) return fail(kUnsupported, "MATMUL: the split-operand tcgen05 form needs unbatched f32 A (K contiguous), B (K or N contiguous) and C (N contiguous)");
        return kOk;
    }
    if (kernel != DFGPU_MATMUL_FFMA && !matmul_umma_supported(p, kernel))
        return fail(kUnsupported, "MATMUL: the requested tcgen05 kernel does not cover this shape, layout or type");
    return kOk;
}

}  // namespace
}  // namespace dfgpu

using namespace dfgpu;

extern "C" int dfgpu_query_matmul(const dfgpu_matmul_params* p, dfgpu_plan_info* info) {
    if (!p || !info) return fail(kInvalidArgument, "MATMUL: null params");
    MatmulArgs g;
    dfgpu_matmul_params copy = *p;
    copy.epilogue_count = 0;
    int status = build_args(copy, nullptr, g);
    if (status) return status;
    int kernel;
    status = choose_kernel(*p, kernel);
    if (status) return status;
    info->kernel = kernel;
    info->launches = 1;
    info->scratch_bytes = 0;
    if (kernel == DFGPU_MATMUL_UMMA_F32X3) {
        SplitMatmul split;
        f32_split_matmul(*p, split);
        info->launches = 3;
        info->scratch_bytes = split.scratch_bytes;
    }
    return kOk;
}

extern "C" int dfgpu_matmul(const dfgpu_matmul_params* p, void* const* tensors, void* scratch, void* stream_handle) {
    if (!p || !tensors) return fail(kInvalidArgument, "MATMUL: null params");
    if (!tensors[0] || !tensors[1] || !tensors[2]) return fail(kInvalidArgument, "MATMUL: null tensor pointer");
    if ((p->a_scale.rank && !tensors[3]) || (p->b_scale.rank && !tensors[4])) return fail(kInvalidArgument, "MATMUL: null block scale pointer");
    MatmulArgs g;
    int status = build_args(*p, tensors, g);
    if (status) return status;
    int kernel;
    status = choose_kernel(*p, kernel);
    if (status) return status;
    cudaStream_t stream = as_stream(stream_handle);
    // (AUTO: operands off the 16-byte boundary TMA needs are read by the CUDA-core kernel instead)
    if (p->kernel == DFGPU_MATMUL_AUTO && (kernel == DFGPU_MATMUL_UMMA_BF16 || kernel == DFGPU_MATMUL_UMMA_MXF8) &&
        ((reinterpret_cast<uintptr_t>(tensors[0]) | reinterpret_cast<uintptr_t>(tensors[1])) & 15u) != 0)
        kernel = DFGPU_MATMUL_FFMA;
    if (p->kernel == DFGPU_MATMUL_AUTO && kernel == DFGPU_MATMUL_FFMA) {
        // what of the CUDA-core form's work other kernels do faster
        FewRows few;
        if (few_rows_form(*p, few)) {
            if ((reinterpret_cast<uintptr_t>(tensors[1]) & 15u) == 0) return launch_few_rows(few, g, tensors, stream);
            if (matmul_f32_cluster_supported(*p)) kernel = DFGPU_MATMUL_UMMA_F32X3_CLUSTER;
        } else if (matmul_f32_flat(*p, tensors)) {
            kernel = DFGPU_MATMUL_UMMA_F32X3_CLUSTER;
        }
    }
    if (kernel == DFGPU_MATMUL_UMMA_F32X3_CLUSTER) return launch_matmul_f32_cluster(*p, tensors, stream);  // (any f32 pointer: 4-byte alignment is enough)
    if (kernel == DFGPU_MATMUL_UMMA_F32X3) {
        SplitMatmul split;
        if (!f32_split_matmul(*p, split)) return fail(kUnsupported, "MATMUL: the split-operand tcgen05 form does not take this matmul");
        if (!scratch || (reinterpret_cast<uintptr_t>(scratch) & 15u) != 0)
            return fail(kInvalidArgument, "MATMUL: the split-operand tcgen05 form needs its 16-byte aligned scratch (dfgpu_query_matmul gives the size)");
        uint8_t* base = static_cast<uint8_t*>(scratch);
        auto place = [](PieceOperand& o, void* source, uint8_t* pieces) {
            o.source = static_cast<const float*>(source);
            o.pieces = reinterpret_cast<uint16_t*>(pieces);
            o.vector = (reinterpret_cast<uintptr_t>(source) & 15u) == 0 && o.source_ld % 4 == 0 ? 1 : 0;
        };
        place(split.a, tensors[0], base);
        place(split.b, tensors[1], base + split.b_offset);
        int* flags = reinterpret_cast<int*>(base + split.flags_offset);
        status = launch_split3(split.a, split.b, flags, stream);
        if (status) return status;
        split.product.a = split.a.pieces;
        split.product.b = split.b.pieces;
        status = launch_matmul_pieces(*p, split.product, tensors, stream);
        if (status) return status;
        dim3 grid(static_cast<unsigned>(std::min<int64_t>((g.m + 63) / 64, 24)), static_cast<unsigned>(std::min<int64_t>((g.n + 63) / 64, 24)), 1);
        launch_chained(matmul_ffma_kernel, dim3(grid), dim3(256), 0, stream, tensors[0], tensors[1], tensors[2], g, flags, split.flag_count);
        return check_launch("MATMUL");
    }
    if (kernel != DFGPU_MATMUL_FFMA) return launch_matmul_umma(*p, tensors, kernel, stream);
    int64_t batches = 1;
    for (int i = 0; i < g.rank - 2; ++i) batches *= p->c.dim[i];
    if (batches > 65535) return fail(kUnsupported, "MATMUL: more than 65535 batch matrices");
    dim3 grid(static_cast<unsigned>((g.m + 63) / 64), static_cast<unsigned>((g.n + 63) / 64), static_cast<unsigned>(batches));
    launch_chained(matmul_ffma_kernel, dim3(grid), dim3(256), 0, stream, tensors[0], tensors[1], tensors[2], g, nullptr, 0);
    return check_launch("MATMUL");
}
