// f32 operands of a contraction as bf16 pieces for the bf16 tensor cores: six-piece copies, or the three pieces once each.
//
// x = xh + xm + xl and w = wh + wm + wl with bf16 pieces (the leading 8 significant bits, the next 8, the last 8; every
// subtraction that forms them is exact), so x * w = xh*wh + xh*wm + xm*wh + xh*wl + xl*wh + xm*wm up to 2^-24 relative:
// a bf16 contraction over six times the depth, the first operand laid out as [xh | xh | xm | xh | xl | xm] and the
// second as [wh | wm | wh | wl | wh | wm], accumulated in f32 by the tensor cores. (Two pieces and three products stop at
// 2^-16, which fails the reference's acceptance rule 1e-4 + 1e-3 |ref| where |ref| is small.)
// A product with an infinite or NaN factor does not survive the split (inf * 0 where the other factor's lower pieces
// are zero), so every CTA of the split kernel also records whether it saw such a value; the caller launches its
// CUDA-core kernel behind the tensor-core one, which redoes the contraction when any CTA did.
#include <algorithm>

#include "common.cuh"
#include "umma.cuh"

namespace dfgpu {
namespace {

// The three bf16 pieces of v; false (and everything in the first piece) when v is infinite or NaN.
__device__ __forceinline__ bool split_f32(float v, uint32_t (&piece)[3]) {
    const uint32_t bits = __float_as_uint(v);
    if ((bits & 0x7f800000u) == 0x7f800000u) {
        piece[0] = bits >> 16 | ((bits & 0xffffu) != 0u ? 0x40u : 0u);  // (a NaN stays a NaN whatever its low bits were)
        piece[1] = piece[2] = 0u;
        return false;
    }
    uint32_t hi = f32_to_bf16_bits(v);
    if ((hi & 0x7f80u) == 0x7f80u) hi = (hi & 0x8000u) | 0x7f7fu;  // rounded past the largest bf16: keep it finite
    const float rest = v - __uint_as_float(hi << 16);
    const uint32_t mid = f32_to_bf16_bits(rest);
    piece[0] = hi;
    piece[1] = mid;
    piece[2] = f32_to_bf16_bits(rest - __uint_as_float(mid << 16));
    return true;
}

__global__ void __launch_bounds__(256)
split6_f32_kernel(SplitOperand first, SplitOperand second, int* __restrict__ flags) {
    chain_wait();
    chain_release();
    first.source = after_chain(first.source);
    second.source = after_chain(second.source);
    bool finite = true;
    float4 v[4];
    bool live[4], in_second[4];
    int64_t quad[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {  // all four loads in flight before the first is used
        quad[i] = static_cast<int64_t>(blockIdx.x) * kSplitQuadsPerCta + i * 256 + threadIdx.x;
        in_second[i] = quad[i] >= first.quads;
        if (in_second[i]) quad[i] -= first.quads;
        const bool s = in_second[i];
        const int64_t row_quads = s ? second.row_quads : first.row_quads;
        live[i] = quad[i] < (s ? second.quads : first.quads);
        if (live[i]) {
            const int64_t row = quad[i] / row_quads, column = (quad[i] - row * row_quads) * 4;
            v[i] = __ldg(reinterpret_cast<const float4*>((s ? second.source : first.source) + row * (s ? second.source_ld : first.source_ld) + column));
        } else {
            v[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        if (!live[i]) continue;
        uint32_t p0[3], p1[3], p2[3], p3[3];
        finite = split_f32(v[i].x, p0) && finite;
        finite = split_f32(v[i].y, p1) && finite;
        finite = split_f32(v[i].z, p2) && finite;
        finite = split_f32(v[i].w, p3) && finite;
        uint2 piece[3];
#pragma unroll
        for (int j = 0; j < 3; ++j) piece[j] = make_uint2(p0[j] | (p1[j] << 16), p2[j] | (p3[j] << 16));
        const bool s = in_second[i];
        const int64_t row_quads = s ? second.row_quads : first.row_quads;
        const int64_t row = quad[i] / row_quads, column = (quad[i] - row * row_quads) * 4;
        uint16_t* out = (s ? second.pieces : first.pieces) + row * (s ? second.row_stride : first.row_stride) + column;
        const int64_t piece_stride = s ? second.piece_stride : first.piece_stride;
        // first operand: h h m h l m; second operand: h m h l h m
        const int order_first[kSplitPieces] = {0, 0, 1, 0, 2, 1}, order_second[kSplitPieces] = {0, 1, 0, 2, 0, 1};
#pragma unroll
        for (int j = 0; j < kSplitPieces; ++j) *reinterpret_cast<uint2*>(out + j * piece_stride) = s ? piece[order_second[j]] : piece[order_first[j]];
    }
    const int any = __syncthreads_or(finite ? 0 : 1);
    if (threadIdx.x == 0) flags[blockIdx.x] = any;
}

// The three pieces themselves, [3][rows][out_ld], for a kernel that multiplies them pair by pair (umma_matmul.cu). 10 bytes
// of traffic an f32 value against 16 with the six copies. Every thread keeps four float4 groups in flight; a row's last group
// may be short, and the groups of an operand off the 16-byte boundaries are read value by value.
__global__ void __launch_bounds__(256)
split3_f32_kernel(PieceOperand first, PieceOperand second, int* __restrict__ flags) {
    chain_wait();
    chain_release();
    first.source = after_chain(first.source);
    second.source = after_chain(second.source);
    const int total = first.groups + second.groups, step = static_cast<int>(gridDim.x) * 256;
    bool finite = true;
    for (int base = blockIdx.x * 256 + threadIdx.x; base < total; base += 4 * step) {
        float4 v[4];
        int64_t target[4];   // -1: nothing there
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int64_t at = static_cast<int64_t>(base) + static_cast<int64_t>(i) * step;
            target[i] = -1;
            v[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (at >= total) continue;
            const PieceOperand& operand = at < first.groups ? first : second;
            const int group = static_cast<int>(at < first.groups ? at : at - first.groups);
            const int row = static_cast<int>(fast_divide(static_cast<uint32_t>(group), operand.by_row)), column = (group - row * operand.row_groups) * 4;
            const float* source = operand.source + row * operand.source_ld + column;
            const int live = operand.row_length - column;
            target[i] = row * operand.out_ld + column;
            if (operand.vector && live >= 4) {
                v[i] = __ldg(reinterpret_cast<const float4*>(source));
            } else {
                v[i].x = __ldg(source);
                if (live > 1) v[i].y = __ldg(source + 1);
                if (live > 2) v[i].z = __ldg(source + 2);
                if (live > 3) v[i].w = __ldg(source + 3);
            }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            if (target[i] < 0) continue;
            const bool in_first = static_cast<int64_t>(base) + static_cast<int64_t>(i) * step < first.groups;
            uint32_t p0[3], p1[3], p2[3], p3[3];
            finite = split_f32(v[i].x, p0) && finite;
            finite = split_f32(v[i].y, p1) && finite;
            finite = split_f32(v[i].z, p2) && finite;
            finite = split_f32(v[i].w, p3) && finite;
            uint16_t* out = (in_first ? first.pieces : second.pieces) + target[i];
            const int64_t piece = in_first ? first.piece_stride : second.piece_stride;
#pragma unroll
            for (int j = 0; j < 3; ++j) *reinterpret_cast<uint2*>(out + j * piece) = make_uint2(p0[j] | (p1[j] << 16), p2[j] | (p3[j] << 16));
        }
    }
    const int any = __syncthreads_or(finite ? 0 : 1);
    if (threadIdx.x == 0) flags[blockIdx.x] = any;
}

}  // namespace

int piece_flag_count(const PieceOperand& first, const PieceOperand& second) {
    return static_cast<int>(std::min<int64_t>((static_cast<int64_t>(first.groups) + second.groups + 1023) / 1024, 148 * 6));
}

int launch_split3(const PieceOperand& first, const PieceOperand& second, int* flags, cudaStream_t stream) {
    launch_chained(split3_f32_kernel, dim3(piece_flag_count(first, second)), dim3(256), 0, stream, first, second, flags);
    return check_launch("f32 operand split");
}

int split_flag_count(const SplitOperand& first, const SplitOperand& second) {
    return static_cast<int>((first.quads + second.quads + kSplitQuadsPerCta - 1) / kSplitQuadsPerCta);
}

int launch_split6(const SplitOperand& first, const SplitOperand& second, int* flags, cudaStream_t stream) {
    launch_chained(split6_f32_kernel, dim3(split_flag_count(first, second)), dim3(256), 0, stream, first, second, flags);
    return check_launch("f32 operand split");
}

}  // namespace dfgpu
