// POINTWISE nodes that could not be fused into a contraction's epilogue.
// One thread per output element, trailing-axis NumPy broadcast, f32 math.
//
// Every mode of the reference's pointwise_result (lib/Compiler/FoundationalGraph.cpp:2581-2955) goes through
// pointwise_value below: the same expression, one separately rounded f32 operation per step, with CUDA's full-precision
// math functions (see sixteen_bit_activation() for dense 16-bit tensors). Dense tensors of one storage type take the kernel of four
// values per load, also where an operand is broadcast along the leading or the trailing axes (a bias, a mask by rows, a
// scalar); anything else (gaps, other broadcasts, mixed storage types, three inputs, GEN_INDEX) one element per thread,
// where ADD / MUL / SUB / RELU_FWD / IDENTITY keep a kernel with nothing else in it.
#include <algorithm>
#include <type_traits>

#include "common.cuh"

namespace dfgpu {
namespace {

__device__ __forceinline__ int64_t broadcast_offset(const View& t, int out_rank, const int64_t* index) {
    int shift = out_rank - t.rank;
    int64_t offset = 0;
    for (int i = 0; i < t.rank; ++i) offset += (t.dim[i] == 1 ? 0 : index[i + shift]) * t.stride[i];
    return offset;
}

struct PointwiseScalars {
    float relu_lower, relu_upper, relu_slope, elu_alpha, softplus_beta, swish_beta;
    int axis;
};

__host__ __device__ constexpr int input_count(int mode) {
    if (mode < 0 || mode >= DFGPU_PW_MODE_COUNT) return 0;
    if (mode == DFGPU_PW_BINARY_SELECT) return 3;
    switch (mode) {
        case DFGPU_PW_ADD: case DFGPU_PW_MUL: case DFGPU_PW_SUB: case DFGPU_PW_DIV: case DFGPU_PW_ADD_SQUARE:
        case DFGPU_PW_MIN: case DFGPU_PW_MAX: case DFGPU_PW_MOD: case DFGPU_PW_POW:
        case DFGPU_PW_LOGICAL_AND: case DFGPU_PW_LOGICAL_OR:
        case DFGPU_PW_CMP_EQ: case DFGPU_PW_CMP_NEQ: case DFGPU_PW_CMP_GT: case DFGPU_PW_CMP_GE: case DFGPU_PW_CMP_LT: case DFGPU_PW_CMP_LE:
        case DFGPU_PW_RELU_BWD: case DFGPU_PW_TANH_BWD: case DFGPU_PW_SIGMOID_BWD: case DFGPU_PW_ELU_BWD:
        case DFGPU_PW_SOFTPLUS_BWD: case DFGPU_PW_SWISH_BWD: case DFGPU_PW_GELU_BWD: case DFGPU_PW_GELU_APPROX_TANH_BWD:
            return 2;
        default: return 1;
    }
}

inline bool simple_mode(int mode) { return mode >= DFGPU_PW_ADD && mode <= DFGPU_PW_SUB; }

// 1 / (1 + exp(-v)) (FoundationalGraph.cpp:2569-2579)
__device__ __forceinline__ float sigmoid_value(float v) { return __fdiv_rn(1.0f, __fadd_rn(1.0f, expf(-v))); }

// ---- activations whose result is rounded to 16 bits ----------------------------------------------------------------
// With erff, tanhf and divisions the instructions set the pace instead of the bytes (GELU_BWD on 33.5 M bf16 values: 55.8 us
// against 30.7 for its bytes). The forms here are one expf and one reciprocal each, arranged so that nothing cancels: errors of a
// few 2^-23 relative over the whole range, tails and zeros included, subnormal results kept. Against the full-precision
// formulas every mode's largest error over all 16-bit inputs, in units of the result's rounding, is no larger.
__device__ __forceinline__ float reciprocal_of_one_or_more(float v) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v));
    return r;
}
__device__ __forceinline__ float exp2_flushing(float v) {
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v));
    return r;
}
// s = 1 / (1 + e^-z) and its complement c = 1 - s, both to f32's relative accuracy.
__device__ __forceinline__ void logistic(float z, float& s, float& c) {
    const float e = expf(-fabsf(z)), larger = reciprocal_of_one_or_more(1.0f + e), smaller = e * larger;
    s = z < 0.0f ? smaller : larger;
    c = z < 0.0f ? larger : smaller;
}
// u: the activation's input, x: the gradient of a _BWD mode. False: not one of these modes.
__device__ __forceinline__ bool sixteen_bit_activation(int mode, float x, float u, const PointwiseScalars& s, float& result) {
    float p, q;
    switch (mode) {
        case DFGPU_PW_SIGMOID_FWD: logistic(u, p, q); result = p; return true;
        case DFGPU_PW_SIGMOID_BWD: logistic(u, p, q); result = x * (p * q); return true;
        case DFGPU_PW_SOFTPLUS_BWD: logistic(s.softplus_beta * u, p, q); result = x * p; return true;
        case DFGPU_PW_SWISH_FWD: logistic(s.swish_beta * u, p, q); result = u * p; return true;
        case DFGPU_PW_SWISH_BWD: {
            const float z = s.swish_beta * u;
            logistic(z, p, q);
            result = x * fmaf(z, p * q, p);
            return true;
        }
        case DFGPU_PW_TANH_FWD: {
            // (1 - e) / (1 + e), e = e^-2|v| (beside 1, e may be flushed); where that cancels, an odd polynomial of least relative error
            // (4e-8 up to 0.35)
            const float e = exp2_flushing(-2.8853900817779268f * fabsf(u)), far = copysignf((1.0f - e) * reciprocal_of_one_or_more(1.0f + e), u), square = u * u;
            const float near = u * fmaf(square, fmaf(square, fmaf(square, -0.0491485f, 0.13299825f), -0.33332663f), 1.0f);
            result = fabsf(u) < 0.35f ? near : far;
            return true;
        }
        case DFGPU_PW_TANH_BWD: logistic(2.0f * u, p, q); result = x * (4.0f * (p * q)); return true;   // 1 - tanh^2
        case DFGPU_PW_GELU_APPROX_TANH_FWD: case DFGPU_PW_GELU_APPROX_TANH_BWD: {   // (1 + tanh t) / 2 = logistic(2 t)
            const float square = u * u, twice = 1.5957691216057308f * fmaf(0.044715f * square, u, u);
            logistic(twice, p, q);
            if (mode == DFGPU_PW_GELU_APPROX_TANH_FWD) {
                result = u * p;
            } else {   // p + u p', p' = p (1 - p) (2 t)'
                const float slope = 1.5957691216057308f * fmaf(0.134145f, square, 1.0f);
                result = x * fmaf(u, slope * (p * q), p);
            }
            return true;
        }
        default: return false;
    }
}

// GELU on two values at once: its polynomial makes it the longest, and the FMA pipe takes pairs of f32.
__device__ __forceinline__ uint64_t pack2(float lo, float hi) {
    uint64_t v;
    asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(lo), "f"(hi));
    return v;
}
__device__ __forceinline__ uint64_t both(float v) { return pack2(v, v); }
__device__ __forceinline__ void unpack2(uint64_t v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
    uint64_t d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
// The upper tail of the normal distribution at |v| over its bell e^(-v^2/2), half of erfc(z) e^(z^2) at z = |v| / sqrt 2, as a
// polynomial in k = 1 / (1 + 0.27 |v|) without constant term: least relative error up to |v| = 14.6, where the bell ends (2.4e-8;
// 3.5e-7 with the rounding of its evaluation).
__device__ __forceinline__ uint64_t tail_over_bell(uint64_t magnitude) {
    float lo, hi;
    unpack2(fma2(both(0.27f), magnitude, both(1.0f)), lo, hi);
    const uint64_t k = pack2(reciprocal_of_one_or_more(lo), reciprocal_of_one_or_more(hi));
    uint64_t sum = both(0.0289688222f);
    sum = fma2(sum, k, both(-0.126524672f));
    sum = fma2(sum, k, both(0.169869289f));
    sum = fma2(sum, k, both(-0.0693096891f));
    sum = fma2(sum, k, both(0.107896969f));
    sum = fma2(sum, k, both(0.0720177665f));
    sum = fma2(sum, k, both(0.101819173f));
    sum = fma2(sum, k, both(0.107541606f));
    sum = fma2(sum, k, both(0.107720733f));
    return mul2(sum, k);
}
template <bool BACKWARD>
__device__ __forceinline__ void sixteen_bit_gelu(const float* x, const float* u, float* result) {
    const uint64_t value = pack2(u[0], u[1]), magnitude = pack2(fabsf(u[0]), fabsf(u[1]));
    float e0, e1;
    unpack2(mul2(mul2(value, value), both(-0.72134752044448170f)), e0, e1);   // (squares of 16-bit values are exact)
    asm("ex2.approx.f32 %0, %0;" : "+f"(e0));
    asm("ex2.approx.f32 %0, %0;" : "+f"(e1));
    const uint64_t bell = pack2(e0, e1), tail = tail_over_bell(magnitude);
    // the distribution function, or its derivative's cdf + u pdf: below zero `below`, above it one less that
    const uint64_t below = BACKWARD ? mul2(bell, fma2(both(-0.3989422804014327f), magnitude, tail)) : mul2(bell, tail);
    float below0, below1, above0, above1;
    unpack2(fma2(below, both(1.0f), both(0.0f)), below0, below1);   // (+0.0: the formula's sum is never -0.0)
    unpack2(fma2(below, both(-1.0f), both(1.0f)), above0, above1);
    unpack2(mul2(BACKWARD ? pack2(x[0], x[1]) : value, pack2(u[0] >= 0.0f ? above0 : below0, u[1] >= 0.0f ? above1 : below1)), result[0], result[1]);
}

// x, y, z: IN_0, IN_1, IN_2 (0 where the mode has none). u: the activation's input (IN_1 of a _BWD mode, else IN_0).
template <bool EXACT>
__device__ __forceinline__ float pointwise_value(int mode, float x, float y, float z, const PointwiseScalars& s, int64_t position) {
    const float u = (mode >= DFGPU_PW_RELU_BWD && input_count(mode) == 2) ? y : x;
    if constexpr (!EXACT) {
        float result;
        if (sixteen_bit_activation(mode, x, u, s, result)) return result;
    }
    switch (mode) {
        case DFGPU_PW_ADD: return __fadd_rn(x, y);
        case DFGPU_PW_MUL: return __fmul_rn(x, y);
        case DFGPU_PW_SUB: return __fsub_rn(x, y);
        case DFGPU_PW_DIV: return __fdiv_rn(x, y);
        case DFGPU_PW_ADD_SQUARE: return __fadd_rn(x, __fmul_rn(y, y));
        case DFGPU_PW_MIN: return minimum_nan(x, y);
        case DFGPU_PW_MAX: return maximum_nan(x, y);
        case DFGPU_PW_MOD: return fmodf(x, y);
        case DFGPU_PW_POW: return powf(x, y);
        case DFGPU_PW_SQRT: return __fsqrt_rn(x);
        case DFGPU_PW_RSQRT: return __fdiv_rn(1.0f, __fsqrt_rn(x));
        case DFGPU_PW_EXP: return expf(x);
        case DFGPU_PW_LOG: return logf(x);
        case DFGPU_PW_NEG: return -x;
        case DFGPU_PW_ABS: return fabsf(x);
        case DFGPU_PW_CEIL: return ceilf(x);
        case DFGPU_PW_FLOOR: return floorf(x);
        case DFGPU_PW_COS: return cosf(x);
        case DFGPU_PW_SIN: return sinf(x);
        case DFGPU_PW_TAN: return tanf(x);
        case DFGPU_PW_ERF: return erff(x);
        case DFGPU_PW_RECIPROCAL: return __fdiv_rn(1.0f, x);
        case DFGPU_PW_IDENTITY: return x;
        case DFGPU_PW_GEN_INDEX: return __ull2float_rn(static_cast<unsigned long long>(position));
        case DFGPU_PW_LOGICAL_NOT: return x == 0.0f ? 1.0f : 0.0f;
        case DFGPU_PW_LOGICAL_AND: return (x != 0.0f) && (y != 0.0f) ? 1.0f : 0.0f;
        case DFGPU_PW_LOGICAL_OR: return (x != 0.0f) || (y != 0.0f) ? 1.0f : 0.0f;
        case DFGPU_PW_BINARY_SELECT: return z != 0.0f ? y : x;
        case DFGPU_PW_CMP_EQ: return x == y ? 1.0f : 0.0f;
        case DFGPU_PW_CMP_NEQ: return x != y ? 1.0f : 0.0f;
        case DFGPU_PW_CMP_GT: return x > y ? 1.0f : 0.0f;
        case DFGPU_PW_CMP_GE: return x >= y ? 1.0f : 0.0f;
        case DFGPU_PW_CMP_LT: return x < y ? 1.0f : 0.0f;
        case DFGPU_PW_CMP_LE: return x <= y ? 1.0f : 0.0f;
        case DFGPU_PW_RELU_FWD: return relu_forward(x, s.relu_lower, s.relu_upper, s.relu_slope);
        case DFGPU_PW_RELU_BWD: return __fmul_rn(x, y < s.relu_lower ? s.relu_slope : (y > s.relu_upper ? 0.0f : 1.0f));
        case DFGPU_PW_TANH_FWD: return tanhf(u);
        case DFGPU_PW_TANH_BWD: { float t = tanhf(u); return __fmul_rn(x, __fsub_rn(1.0f, __fmul_rn(t, t))); }
        case DFGPU_PW_SIGMOID_FWD: return sigmoid_value(u);
        case DFGPU_PW_SIGMOID_BWD: { float v = sigmoid_value(u); return __fmul_rn(x, __fmul_rn(v, __fsub_rn(1.0f, v))); }
        case DFGPU_PW_ELU_FWD: { float e = expf(u); return u >= 0.0f ? u : __fmul_rn(s.elu_alpha, __fsub_rn(e, 1.0f)); }
        case DFGPU_PW_ELU_BWD: { float e = expf(u); return __fmul_rn(x, u >= 0.0f ? 1.0f : __fmul_rn(s.elu_alpha, e)); }
        case DFGPU_PW_SOFTPLUS_FWD: {
            float scaled = __fmul_rn(s.softplus_beta, u);
            float logarithm = logf(__fadd_rn(1.0f, expf(-fabsf(scaled))));
            return __fdiv_rn(__fadd_rn(maximum_nan(scaled, 0.0f), logarithm), s.softplus_beta);
        }
        case DFGPU_PW_SOFTPLUS_BWD: return __fmul_rn(x, sigmoid_value(__fmul_rn(s.softplus_beta, u)));
        case DFGPU_PW_SWISH_FWD: return __fmul_rn(u, sigmoid_value(__fmul_rn(s.swish_beta, u)));
        case DFGPU_PW_SWISH_BWD: {
            float scaled = __fmul_rn(s.swish_beta, u);
            float v = sigmoid_value(scaled);
            return __fmul_rn(x, __fadd_rn(v, __fmul_rn(scaled, __fmul_rn(v, __fsub_rn(1.0f, v)))));
        }
        case DFGPU_PW_GELU_FWD: case DFGPU_PW_GELU_BWD: {
            float cdf = __fmul_rn(0.5f, __fadd_rn(1.0f, erff(__fmul_rn(u, 0.7071067811865475f))));
            if (mode == DFGPU_PW_GELU_FWD) return __fmul_rn(u, cdf);
            float density = __fmul_rn(0.3989422804014327f, expf(__fmul_rn(-0.5f, __fmul_rn(u, u))));
            return __fmul_rn(x, __fadd_rn(cdf, __fmul_rn(u, density)));
        }
        case DFGPU_PW_GELU_APPROX_TANH_FWD: case DFGPU_PW_GELU_APPROX_TANH_BWD: {
            float square = __fmul_rn(u, u);
            float cubic = __fmul_rn(square, u);
            float inner = __fmul_rn(0.7978845608028654f, __fadd_rn(u, __fmul_rn(0.044715f, cubic)));
            float t = tanhf(inner);
            float cdf = __fmul_rn(0.5f, __fadd_rn(1.0f, t));
            if (mode == DFGPU_PW_GELU_APPROX_TANH_FWD) return __fmul_rn(u, cdf);
            float inner_derivative = __fmul_rn(0.7978845608028654f, __fadd_rn(1.0f, __fmul_rn(0.134145f, square)));
            float tanh_derivative = __fsub_rn(1.0f, __fmul_rn(t, t));
            return __fmul_rn(x, __fadd_rn(cdf, __fmul_rn(0.5f, __fmul_rn(u, __fmul_rn(tanh_derivative, inner_derivative)))));
        }
        default: return x;
    }
}

// Four neighbouring values of a dense tensor of type T.
template <typename T, int MODE>
__device__ __forceinline__ void four_values(const float (&x)[4], const float (&y)[4], const PointwiseScalars& s, float (&r)[4]) {
    if constexpr (sizeof(T) == 2 && (MODE == DFGPU_PW_GELU_FWD || MODE == DFGPU_PW_GELU_BWD)) {
#pragma unroll
        for (int j = 0; j < 4; j += 2) sixteen_bit_gelu<MODE == DFGPU_PW_GELU_BWD>(x + j, (MODE == DFGPU_PW_GELU_BWD ? y : x) + j, r + j);
    } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) r[j] = pointwise_value<sizeof(T) == 4>(MODE, x[j], y[j], 0.0f, s, 0);
    }
}

// Any mode, any strides and storage types: one thread per output element.
__global__ void pointwise_general_kernel(const void* a, const void* b, const void* c, void* out, View av, View bv, View cv, View ov,
                                         int mode, PointwiseScalars s, int64_t total) {
    chain_begin();
    int64_t flat = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (flat >= total) return;
    int64_t index[DFGPU_MAX_RANK];
    int64_t out_offset = 0;
    for (int i = ov.rank - 1; i >= 0; --i) {
        index[i] = flat % ov.dim[i];
        flat /= ov.dim[i];
        out_offset += index[i] * ov.stride[i];
    }
    const int inputs = input_count(mode);
    float x = load_as_f32(a, av.dtype, broadcast_offset(av, ov.rank, index));
    float y = inputs >= 2 ? load_as_f32(b, bv.dtype, broadcast_offset(bv, ov.rank, index)) : 0.0f;
    float z = inputs >= 3 ? load_as_f32(c, cv.dtype, broadcast_offset(cv, ov.rank, index)) : 0.0f;
    int64_t position = mode == DFGPU_PW_GEN_INDEX ? index[s.axis] : 0;
    store_from_f32(out, ov.dtype, out_offset, pointwise_value<true>(mode, x, y, z, s, position));
}

__global__ void pointwise_kernel(const void* a, const void* b, void* out, View av, View bv, View ov, int mode,
                                 float lower, float upper, float slope, int64_t total) {
    chain_begin();
    int64_t flat = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (flat >= total) return;
    int64_t index[DFGPU_MAX_RANK];
    int64_t out_offset = 0;
    for (int i = ov.rank - 1; i >= 0; --i) {
        index[i] = flat % ov.dim[i];
        flat /= ov.dim[i];
        out_offset += index[i] * ov.stride[i];
    }
    float x = load_as_f32(a, av.dtype, broadcast_offset(av, ov.rank, index));
    float y = 0.0f;
    if (mode == DFGPU_PW_ADD || mode == DFGPU_PW_MUL || mode == DFGPU_PW_SUB)
        y = load_as_f32(b, bv.dtype, broadcast_offset(bv, ov.rank, index));
    float result;
    switch (mode) {
        case DFGPU_PW_ADD: result = __fadd_rn(x, y); break;
        case DFGPU_PW_MUL: result = __fmul_rn(x, y); break;
        case DFGPU_PW_SUB: result = __fsub_rn(x, y); break;
        case DFGPU_PW_RELU_FWD: result = relu_forward(x, lower, upper, slope); break;
        default: result = x; break;
    }
    store_from_f32(out, ov.dtype, out_offset, result);
}

// All operands packed with identical dims: quads of four values. A quad is loaded as it is stored (16 bytes of f32, 8 of
// bf16) and widened only where it is used, so that the quads a thread has in flight cost a register per 4 bytes.
template <typename T> struct Quad;
template <> struct Quad<float> { using type = float4; };
template <> struct Quad<__nv_bfloat16> { using type = uint2; };
template <> struct Quad<__half> { using type = ushort4; };  // (a type of its own, so that widen() tells HALF from BFLOAT16)

template <typename T>
__device__ __forceinline__ typename Quad<T>::type load_quad(const void* p, int64_t i) {
    return __ldg(reinterpret_cast<const typename Quad<T>::type*>(static_cast<const T*>(p) + i));
}
__device__ __forceinline__ void widen(const float4& r, float (&v)[4]) { v[0] = r.x; v[1] = r.y; v[2] = r.z; v[3] = r.w; }
__device__ __forceinline__ void widen(const uint2& r, float (&v)[4]) {
    v[0] = __uint_as_float(r.x << 16); v[1] = __uint_as_float(r.x & 0xffff0000u);
    v[2] = __uint_as_float(r.y << 16); v[3] = __uint_as_float(r.y & 0xffff0000u);
}
__device__ __forceinline__ void widen(const ushort4& r, float (&v)[4]) {
    v[0] = __half2float(__ushort_as_half(r.x)); v[1] = __half2float(__ushort_as_half(r.y));
    v[2] = __half2float(__ushort_as_half(r.z)); v[3] = __half2float(__ushort_as_half(r.w));
}
template <typename T>
__device__ __forceinline__ void store4(void* p, int64_t i, const float (&v)[4]);
template <>
__device__ __forceinline__ void store4<float>(void* p, int64_t i, const float (&v)[4]) {
    *reinterpret_cast<float4*>(static_cast<float*>(p) + i) = make_float4(v[0], v[1], v[2], v[3]);
}
template <>
__device__ __forceinline__ void store4<__nv_bfloat16>(void* p, int64_t i, const float (&v)[4]) {
    __nv_bfloat162 lo = __floats2bfloat162_rn(v[0], v[1]), hi = __floats2bfloat162_rn(v[2], v[3]);  // the same rounding, two values per cvt
    *reinterpret_cast<uint2*>(static_cast<uint16_t*>(p) + i) = make_uint2(*reinterpret_cast<uint32_t*>(&lo), *reinterpret_cast<uint32_t*>(&hi));
}

// Quads of four values a thread keeps in flight: its U quads lie one block-width apart, so that each of a warp's loads
// stays contiguous; every load is issued before the first value is used. 32 bytes per thread and operand: with 8 (bf16)
// or 16 (f32) the loads in flight of a full SM do not cover the latency of HBM.
template <>
__device__ __forceinline__ void store4<__half>(void* p, int64_t i, const float (&v)[4]) {
    __half2 lo = __floats2half2_rn(v[0], v[1]), hi = __floats2half2_rn(v[2], v[3]);
    *reinterpret_cast<uint2*>(static_cast<uint16_t*>(p) + i) = make_uint2(*reinterpret_cast<uint32_t*>(&lo), *reinterpret_cast<uint32_t*>(&hi));
}

// Eight values of a 16-bit type.
template <typename T>
__device__ __forceinline__ void store8(void* p, int64_t i, const float (&v)[2][4]) {
    uint32_t words[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const float lo = v[j >> 1][2 * (j & 1)], hi = v[j >> 1][2 * (j & 1) + 1];
        if constexpr (std::is_same_v<T, __nv_bfloat16>) {
            const __nv_bfloat162 two = __floats2bfloat162_rn(lo, hi);
            words[j] = *reinterpret_cast<const uint32_t*>(&two);
        } else {
            const __half2 two = __floats2half2_rn(lo, hi);
            words[j] = *reinterpret_cast<const uint32_t*>(&two);
        }
    }
    *reinterpret_cast<uint4*>(static_cast<uint16_t*>(p) + i) = make_uint4(words[0], words[1], words[2], words[3]);
}

template <typename T> struct QuadsInFlight;
template <> struct QuadsInFlight<float> { static constexpr int value = 2; };
template <> struct QuadsInFlight<__nv_bfloat16> { static constexpr int value = 4; };
template <> struct QuadsInFlight<__half> { static constexpr int value = 4; };

constexpr int kPackedThreads = 256;
// CTAs per SM of the dense kernel that walk the tiles between them, in eights, where a CTA gets two tiles at most: 4096 x 3072 bf16 and a bias, 3072 tiles, 10.3 us
// with a CTA each (fours), 9.1 so; RELU of 4097 x 3071 10.4 and 9.5. Beyond that the walks drift apart in memory and a CTA a tile is faster:
// TANH of 13747 x 3007 bf16 30.4 walking, 27.2; and so it is in fours from the start: 16384 x 4100 bf16 and a bias 55 walking, 42.5, f32 TANH of
// 13747 x 3007 54.6 and 49.2.
constexpr unsigned kDenseBlocks = 16;

template <typename T>
unsigned packed_grid(int64_t total) {
    const int64_t per_block = static_cast<int64_t>(kPackedThreads) * 4 * QuadsInFlight<T>::value;
    return static_cast<unsigned>((total + per_block - 1) / per_block);
}

// Every mode with one or two inputs (not GEN_INDEX, which needs the element's index). The mode is looked at once per
// thread: the switch leads into a body compiled for that mode alone. A switch per value made every mode cost ~50 us on
// 25.7 M values whatever its arithmetic, and even a five-way switch per value held bf16 RELU_FWD at 37 us (23 us here).
template <typename T, int MODE>
__device__ __forceinline__ void packed_body(const void* a, const void* b, void* out, const PointwiseScalars& s, int64_t total) {
    constexpr int U = QuadsInFlight<T>::value;
    constexpr bool binary = input_count(MODE) == 2;
    const int64_t first = (static_cast<int64_t>(blockIdx.x) * U * kPackedThreads + threadIdx.x) * 4;
    chain_wait();
    a = after_chain(a);
    b = after_chain(b);
    typename Quad<T>::type raw_x[U], raw_y[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const int64_t i = first + static_cast<int64_t>(u) * kPackedThreads * 4;
        if (i < total) {
            raw_x[u] = load_quad<T>(a, i);
            if (binary) raw_y[u] = load_quad<T>(b, i);
        }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const int64_t i = first + static_cast<int64_t>(u) * kPackedThreads * 4;
        if (i >= total) break;
        float x[4], y[4] = {0.0f, 0.0f, 0.0f, 0.0f}, r[4];
        widen(raw_x[u], x);
        if (binary) widen(raw_y[u], y);
        four_values<T, MODE>(x, y, s, r);
        store4<T>(out, i, r);
    }
}

#define DFGPU_PW_EVERY_MODE(X)                                                                                              \
    X(0) X(1) X(2) X(3) X(4) X(5) X(6) X(7) X(8) X(9) X(10) X(11) X(12) X(13) X(14) X(15) X(16) X(17) X(18) X(19) X(20) X(21) \
    X(22) X(23) X(24) X(25) X(26) X(27) X(28) X(29) X(30) X(31) X(32) X(33) X(34) X(35) X(36) X(37) X(38) X(39) X(40) X(41)  \
    X(42) X(43) X(44) X(45) X(46) X(47) X(48) X(49)
static_assert(DFGPU_PW_MODE_COUNT == 50, "DFGPU_PW_EVERY_MODE lists every mode");

// One kernel for the modes with one input and one for those with two. 32 registers, a full SM of 2048 threads, cover
// the latency of HBM best (bf16 RELU_FWD: 84 % of the copy bandwidth against 76 % at 48 registers) except for two bf16
// inputs, where eight quads in flight per thread want 48 registers (92 % against 88 % when held to 32).
template <typename T, int INPUTS>
__global__ void __launch_bounds__(kPackedThreads, (sizeof(T) == 2 && INPUTS == 2) ? 5 : 2048 / kPackedThreads)
pointwise_general_packed_kernel(const void* a, const void* b, void* out, int mode, PointwiseScalars s, int64_t total) {
    chain_release();
    switch (mode) {   // (each body waits for the kernel before: see dense_body())
#define DFGPU_PW_CASE(M) case M: if constexpr (input_count(M) == INPUTS) packed_body<T, M>(a, b, out, s, total); break;
        DFGPU_PW_EVERY_MODE(DFGPU_PW_CASE)
#undef DFGPU_PW_CASE
        default: break;
    }
}

// ---- dense tensors with broadcast operands, any count and pointer ------------------------------------------------
// The output is dense in some order of its axes; an operand has the same order (FULL), only the innermost axes (PERIOD: a bias
// along the channels), only the outermost ones (REPEAT: a value per row, or one for all), and is indexed by one division per
// quad. Where rows or pointers do not fall on quads the same kernel goes value by value. 4096 x 3072 bf16 + bias: 118 us
// with an index computation per value and axis.
enum { kFull = 0, kPeriod = 1, kRepeat = 2 };
struct DenseOperand {
    const void* data;
    int32_t kind;
    int32_t vector;       // neighbouring values of this operand (or of what they repeat) that may be read at once: 8 (16-bit types), 4, or 0
    FastDivisor by;       // PERIOD: values before it starts again; REPEAT: outputs per value
};

template <typename T>
__device__ __forceinline__ float one_value(const void* p, uint32_t i) {
    if constexpr (sizeof(T) == 4) return __ldg(static_cast<const float*>(p) + i);
    const uint16_t bits = __ldg(static_cast<const uint16_t*>(p) + i);
    if constexpr (std::is_same_v<T, __nv_bfloat16>) return __uint_as_float(static_cast<uint32_t>(bits) << 16);
    return __half2float(__ushort_as_half(bits));
}
__device__ __forceinline__ uint32_t dense_index(const DenseOperand& o, uint32_t i) {
    if (o.kind == kFull) return i;
    const uint32_t q = fast_divide(i, o.by);
    return o.kind == kRepeat ? q : i - q * o.by.divisor;
}
// WIDTH values, or the one value they repeat, as they are stored: nothing waits for them before widen_raw().
template <typename T, int WIDTH> struct Raw { uint32_t words[WIDTH * sizeof(T) / 4]; };
template <typename T, int WIDTH>
__device__ __forceinline__ Raw<T, WIDTH> load_one(const DenseOperand& o, uint32_t index) {
    Raw<T, WIDTH> raw{};
    const T* p = static_cast<const T*>(o.data) + index;
    if constexpr (sizeof(T) == 4) raw.words[0] = __ldg(reinterpret_cast<const uint32_t*>(p));
    else raw.words[0] = __ldg(reinterpret_cast<const uint16_t*>(p));
    return raw;
}
template <typename T, int WIDTH>
__device__ __forceinline__ Raw<T, WIDTH> load_run(const DenseOperand& o, uint32_t index) {
    Raw<T, WIDTH> raw;
    const T* p = static_cast<const T*>(o.data) + index;
    if constexpr (sizeof(raw) == 16) {
        const uint4 v = __ldg(reinterpret_cast<const uint4*>(p));
        raw.words[0] = v.x, raw.words[1] = v.y, raw.words[2] = v.z, raw.words[3] = v.w;
    } else {
        const uint2 v = __ldg(reinterpret_cast<const uint2*>(p));
        raw.words[0] = v.x, raw.words[1] = v.y;
    }
    return raw;
}
template <typename T, int WIDTH>
__device__ __forceinline__ Raw<T, WIDTH> load_raw(const DenseOperand& o, uint32_t i) {
    const uint32_t index = dense_index(o, i);
    return o.kind == kRepeat ? load_one<T, WIDTH>(o, index) : load_run<T, WIDTH>(o, index);
}
// Values 4 * quad ... 4 * quad + 3 of them.
template <typename T, int WIDTH>
__device__ __forceinline__ void widen_raw(const DenseOperand& o, const Raw<T, WIDTH>& raw, int quad, float (&v)[4]) {
    if constexpr (sizeof(T) == 4) {
#pragma unroll
        for (int j = 0; j < 4; ++j) v[j] = __uint_as_float(raw.words[j]);
    } else {
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const uint32_t two = raw.words[2 * quad + j];
            if constexpr (std::is_same_v<T, __nv_bfloat16>) {
                v[2 * j] = __uint_as_float(two << 16);
                v[2 * j + 1] = __uint_as_float(two & 0xffff0000u);
            } else {
                const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&two));
                v[2 * j] = f.x;
                v[2 * j + 1] = f.y;
            }
        }
    }
    if (o.kind == kRepeat) {
        float one = v[0];
        if constexpr (sizeof(T) == 2)
            if (quad > 0) {   // (the one value lies in the first word)
                if constexpr (std::is_same_v<T, __nv_bfloat16>) one = __uint_as_float(raw.words[0] << 16);
                else one = __low2float(*reinterpret_cast<const __half2*>(&raw.words[0]));
            }
        v[0] = v[1] = v[2] = v[3] = one;
    }
}
template <typename T>
__device__ __forceinline__ void load_dense(const DenseOperand& o, uint32_t i, uint32_t total, float (&v)[4]) {
    if (o.vector && i + 4 <= total) {
        const uint32_t at = dense_index(o, i);
        if (o.kind == kRepeat) v[0] = v[1] = v[2] = v[3] = one_value<T>(o.data, at);
        else widen(load_quad<T>(o.data, at), v);
        return;
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) v[j] = i + j < total ? one_value<T>(o.data, dense_index(o, i + j)) : 0.0f;
}

template <typename T, int MODE, int WIDTH>
__device__ __forceinline__ void dense_tile(const DenseOperand& a, const DenseOperand& b, void* out, const PointwiseScalars& s, uint32_t tile) {
    constexpr int U = QuadsInFlight<T>::value * 4 / WIDTH;
    constexpr bool binary = input_count(MODE) == 2;
    const uint32_t first = tile + threadIdx.x * WIDTH;
    Raw<T, WIDTH> raw_x[U], raw_y[U];
    // Every load is in flight before the first value is used. (In fours of 16 bits an operand's form is looked at once for all of them: with a look
    // before each load 16384 x 4100 bf16 and a bias took 53 us for 42.5. Eights and f32 lose by it, 9.1 -> 9.9 for 4096 x 3072 and 16.4 -> 17.3.)
    if constexpr (sizeof(T) == 2 && WIDTH == 4) {
        auto fetch = [&](const DenseOperand& o, Raw<T, WIDTH> (&raw)[U]) {
            if (o.kind == kRepeat) {
#pragma unroll
                for (int u = 0; u < U; ++u) raw[u] = load_one<T, WIDTH>(o, fast_divide(first + u * kPackedThreads * WIDTH, o.by));
            } else {
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const uint32_t i = first + u * kPackedThreads * WIDTH;
                    raw[u] = load_run<T, WIDTH>(o, o.kind == kFull ? i : i - fast_divide(i, o.by) * o.by.divisor);
                }
            }
        };
        fetch(a, raw_x);
        if (binary) fetch(b, raw_y);
    } else {
#pragma unroll
        for (int u = 0; u < U; ++u) {
            raw_x[u] = load_raw<T, WIDTH>(a, first + u * kPackedThreads * WIDTH);
            if (binary) raw_y[u] = load_raw<T, WIDTH>(b, first + u * kPackedThreads * WIDTH);
        }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
        float r[WIDTH / 4][4];
#pragma unroll
        for (int quad = 0; quad < WIDTH / 4; ++quad) {
            float x[4], y[4] = {0.0f, 0.0f, 0.0f, 0.0f};
            widen_raw<T, WIDTH>(a, raw_x[u], quad, x);
            if (binary) widen_raw<T, WIDTH>(b, raw_y[u], quad, y);
            four_values<T, MODE>(x, y, s, r[quad]);
        }
        if constexpr (WIDTH == 8) store8<T>(out, first + u * kPackedThreads * WIDTH, r);
        else store4<T>(out, first + u * kPackedThreads * WIDTH, r[0]);
    }
}
// WIDTH 8: every operand's and the output's runs are of whole eights. 4: of whole fours (`vector` kAll), or the output's only, or not even those (0).
enum { kOutputOnly = 1, kAll = 2 };
template <typename T, int MODE, int WIDTH, bool WALK>
__device__ __forceinline__ void dense_body(DenseOperand& a, DenseOperand& b, void* out, int vector, const PointwiseScalars& s, uint32_t total) {
    constexpr int U = QuadsInFlight<T>::value;
    constexpr uint32_t kTile = U * kPackedThreads * 4;
    constexpr bool binary = input_count(MODE) == 2;
    chain_wait();   // (here, when the mode's code and the operands' forms are known)
    a.data = after_chain(a.data);
    b.data = after_chain(b.data);
    uint32_t tile = blockIdx.x * kTile;
    if (!WALK && vector == kAll && tile + kTile <= total) return dense_tile<T, MODE, WIDTH>(a, b, out, s, tile);
    do {
        if (WALK && vector == kAll && tile + kTile <= total) {
            dense_tile<T, MODE, WIDTH>(a, b, out, s, tile);
        } else {
            const uint32_t first = tile + threadIdx.x * 4;
#pragma unroll 1
            for (int u = 0; u < U; ++u) {
                const uint32_t i = first + u * kPackedThreads * 4;
                if (i >= total) break;
                float x[4], y[4] = {0.0f, 0.0f, 0.0f, 0.0f}, r[4];
                load_dense<T>(a, i, total, x);
                if (binary) load_dense<T>(b, i, total, y);
                four_values<T, MODE>(x, y, s, r);
                if (vector != 0 && i + 4 <= total) {
                    store4<T>(out, i, r);
                } else {
                    for (int j = 0; j < 4; ++j) {
                        if (i + j >= total) break;
                        if constexpr (sizeof(T) == 4) static_cast<float*>(out)[i + j] = r[j];
                        else if constexpr (std::is_same_v<T, __nv_bfloat16>) static_cast<uint16_t*>(out)[i + j] = f32_to_bf16_bits(r[j]);
                        else static_cast<__half*>(out)[i + j] = __float2half_rn(r[j]);
                    }
                }
            }
        }
        tile += gridDim.x * kTile;
    } while (WALK && tile < total);
}

template <typename T, int INPUTS, int WIDTH, bool WALK>
__global__ void __launch_bounds__(kPackedThreads)
pointwise_dense_kernel(DenseOperand a, DenseOperand b, void* out, int vector, int mode, PointwiseScalars s, uint32_t total) {
    chain_release();
    switch (mode) {   // (each body waits for the kernel before)
#define DFGPU_PW_CASE(M) case M: if constexpr (input_count(M) == INPUTS) dense_body<T, M, WIDTH, WALK>(a, b, out, vector, s, total); break;
        DFGPU_PW_EVERY_MODE(DFGPU_PW_CASE)
#undef DFGPU_PW_CASE
        default: break;
    }
}

// The output's axes from the outermost to the innermost as they lie in memory, or false when there are gaps between them.
bool dense_order(const dfgpu_tensor& out, int (&order)[DFGPU_MAX_RANK], int& count) {
    count = 0;
    for (int i = 0; i < out.rank; ++i)
        if (out.dim[i] != 1) order[count++] = i;
    std::stable_sort(order, order + count, [&](int a, int b) { return out.stride[a] > out.stride[b]; });
    int64_t expected = 1;
    for (int i = count - 1; i >= 0; --i) {
        if (out.stride[order[i]] != expected) return false;
        expected *= out.dim[order[i]];
    }
    return expected < (1ll << 31) - 65536;
}

// Values that may be read or written at once, by the pointer, and at the start of every run of `length` of them.
int vector_of(const void* data, int bytes) {
    const uintptr_t address = reinterpret_cast<uintptr_t>(data);
    return bytes == 2 && address % 16 == 0 ? 8 : (address % (4 * bytes) == 0 ? 4 : 0);
}
int vector_in(int64_t length, int bytes) { return bytes == 2 && length % 8 == 0 ? 8 : (length % 4 == 0 ? 4 : 0); }

bool dense_operand(const dfgpu_tensor& t, const dfgpu_tensor& out, const int (&order)[DFGPU_MAX_RANK], int count, const void* data, DenseOperand& o) {
    const int shift = out.rank - t.rank;
    int64_t inner = 1, own = 1, held = 1;   // outputs and own values so far, from the innermost axis; outputs per own value
    int64_t period = 0;                     // set where the operand's axes end
    for (int i = count - 1; i >= 0; --i) {
        const int axis = order[i] - shift;
        const int64_t extent = out.dim[order[i]];
        if (axis >= 0 && t.dim[axis] == extent && t.stride[axis] == own) {
            if (period != 0) return false;   // (a broadcast axis between its own)
            own *= extent;
        } else if (axis < 0 || t.dim[axis] == 1) {
            if (own == 1) held *= extent;    // a trailing broadcast axis
            else if (period == 0) period = inner;
        } else {
            return false;
        }
        inner *= extent;
    }
    const int bytes = dtype_bytes(t.dtype);
    const int aligned = vector_of(data, bytes);
    o.data = data;
    o.by = make_fast_divisor(1);
    if (held > 1) {
        if (period != 0) return false;
        o.kind = kRepeat;
        o.by = make_fast_divisor(static_cast<uint32_t>(held));
        o.vector = vector_in(held, bytes);
    } else if (period != 0) {
        o.kind = kPeriod;
        o.by = make_fast_divisor(static_cast<uint32_t>(period));
        o.vector = std::min(vector_in(period, bytes), aligned);
    } else {
        o.kind = kFull;
        o.vector = aligned;
    }
    return true;
}

template <typename T>
void launch_dense(int inputs, const DenseOperand& a, const DenseOperand& b, void* out, int mode, const PointwiseScalars& s, int64_t total, cudaStream_t stream) {
    const int out_width = vector_of(out, sizeof(T)), width = std::min(out_width, std::min(a.vector, inputs == 2 ? b.vector : 8));
    const unsigned tiles = packed_grid<T>(total), walkers = kDenseBlocks * static_cast<unsigned>(sm_count());
    auto launch = [&](auto kernel, unsigned grid) {
        launch_chained(kernel, dim3(grid), dim3(kPackedThreads), 0, stream, a, b, out, width != 0 ? kAll : (out_width != 0 ? kOutputOnly : 0), mode, s, static_cast<uint32_t>(total));
    };
    if constexpr (sizeof(T) == 2) {
        if (width == 8 && tiles <= 2 * walkers) return launch(inputs == 1 ? pointwise_dense_kernel<T, 1, 8, true> : pointwise_dense_kernel<T, 2, 8, true>, std::min(tiles, walkers));
        if (width == 8) return launch(inputs == 1 ? pointwise_dense_kernel<T, 1, 8, false> : pointwise_dense_kernel<T, 2, 8, false>, tiles);
    }
    launch(inputs == 1 ? pointwise_dense_kernel<T, 1, 4, false> : pointwise_dense_kernel<T, 2, 4, false>, tiles);
}

template <typename T>
void launch_packed(int inputs, const void* a, const void* b, void* out, int mode, const PointwiseScalars& s, int64_t total, cudaStream_t stream) {
    if (inputs == 1) launch_chained(pointwise_general_packed_kernel<T, 1>, dim3(packed_grid<T>(total)), dim3(kPackedThreads), 0, stream, a, b, out, mode, s, total);
    else launch_chained(pointwise_general_packed_kernel<T, 2>, dim3(packed_grid<T>(total)), dim3(kPackedThreads), 0, stream, a, b, out, mode, s, total);
}

bool same_packed(const dfgpu_tensor& a, const dfgpu_tensor& b) {
    if (a.rank != b.rank) return false;
    for (int i = 0; i < a.rank; ++i)
        if (a.dim[i] != b.dim[i]) return false;
    return is_packed_row_major(a) && is_packed_row_major(b);
}

int validate(const dfgpu_pointwise_params& p, int& inputs) {
    inputs = input_count(p.mode);
    if (inputs == 0) return fail(kUnsupported, "POINTWISE: mode %d is not executable on this backend", p.mode);
    if (!valid_tensor(p.in0) || !valid_tensor(p.out) || (inputs >= 2 && !valid_tensor(p.in1)) || (inputs >= 3 && !valid_tensor(p.in2)))
        return fail(kInvalidShape, "POINTWISE: tensor rank or extent out of range");
    const dfgpu_tensor* operands[3] = {&p.in0, &p.in1, &p.in2};
    for (int n = 0; n < inputs; ++n) {
        const dfgpu_tensor& t = *operands[n];
        if (t.rank > p.out.rank) return fail(kInvalidShape, "POINTWISE: input rank exceeds output rank");
        int shift = p.out.rank - t.rank;
        for (int i = 0; i < t.rank; ++i)
            if (t.dim[i] != 1 && t.dim[i] != p.out.dim[i + shift])
                return fail(kInvalidShape, "POINTWISE: input does not broadcast onto the output");
        if (t.dtype != DFGPU_F32 && t.dtype != DFGPU_BF16 && t.dtype != DFGPU_F16)
            return fail(kUnsupported, "POINTWISE: unsupported input type");
    }
    if (p.out.dtype != DFGPU_F32 && p.out.dtype != DFGPU_BF16 && p.out.dtype != DFGPU_F16)
        return fail(kUnsupported, "POINTWISE: unsupported output type");
    if (p.mode == DFGPU_PW_GEN_INDEX && (p.axis < 0 || p.axis >= p.out.rank))
        return fail(kInvalidValue, "POINTWISE: GEN_INDEX needs an axis inside the output's rank");
    if ((p.mode == DFGPU_PW_SOFTPLUS_FWD || p.mode == DFGPU_PW_SOFTPLUS_BWD) && !(p.softplus_beta > 0.0f))
        return fail(kInvalidValue, "POINTWISE: softplus beta must be positive");
    if ((p.mode == DFGPU_PW_RELU_FWD || p.mode == DFGPU_PW_RELU_BWD) && p.relu_lower > p.relu_upper)
        return fail(kInvalidValue, "POINTWISE: ReLU lower clip exceeds upper clip");
    return kOk;
}

}  // namespace
}  // namespace dfgpu

using namespace dfgpu;

extern "C" int dfgpu_pointwise_input_count(int32_t mode) { return input_count(mode); }

extern "C" int dfgpu_query_pointwise(const dfgpu_pointwise_params* p, dfgpu_plan_info* info) {
    if (!p || !info) return fail(kInvalidArgument, "POINTWISE: null params");
    int inputs;
    int status = validate(*p, inputs);
    if (status) return status;
    info->kernel = 1;
    info->launches = 1;
    info->scratch_bytes = 0;
    return kOk;
}

extern "C" int dfgpu_pointwise(const dfgpu_pointwise_params* p, void* const* tensors, void* scratch, void* stream_handle) {
    (void)scratch;
    if (!p || !tensors) return fail(kInvalidArgument, "POINTWISE: null params");
    int inputs;
    int status = validate(*p, inputs);
    if (status) return status;
    const bool binary = inputs == 2;
    if (!tensors[0] || !tensors[2] || (inputs >= 2 && !tensors[1]) || (inputs >= 3 && !tensors[3]))
        return fail(kInvalidArgument, "POINTWISE: null tensor pointer");
    cudaStream_t stream = as_stream(stream_handle);
    int64_t total = element_count(p->out);
    auto aligned16 = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15u) == 0; };
    bool packed = same_packed(p->in0, p->out) && (!binary || same_packed(p->in1, p->out)) && total % 4 == 0 &&
                  aligned16(tensors[0]) && aligned16(tensors[2]) && (!binary || aligned16(tensors[1]));
    bool f32_all = p->in0.dtype == DFGPU_F32 && p->out.dtype == DFGPU_F32 && (!binary || p->in1.dtype == DFGPU_F32);
    bool bf16_all = p->in0.dtype == DFGPU_BF16 && p->out.dtype == DFGPU_BF16 && (!binary || p->in1.dtype == DFGPU_BF16);
    bool f16_all = p->in0.dtype == DFGPU_F16 && p->out.dtype == DFGPU_F16 && (!binary || p->in1.dtype == DFGPU_F16);
    PointwiseScalars s{p->relu_lower, p->relu_upper, p->relu_slope, p->elu_alpha, p->softplus_beta, p->swish_beta, p->axis};
    if (packed && (f32_all || bf16_all || f16_all) && inputs <= 2 && p->mode != DFGPU_PW_GEN_INDEX) {
        if (f32_all) launch_packed<float>(inputs, tensors[0], tensors[1], tensors[2], p->mode, s, total, stream);
        else if (f16_all) launch_packed<__half>(inputs, tensors[0], tensors[1], tensors[2], p->mode, s, total, stream);
        else launch_packed<__nv_bfloat16>(inputs, tensors[0], tensors[1], tensors[2], p->mode, s, total, stream);
        return check_launch("POINTWISE");
    }
    if ((f32_all || bf16_all || f16_all) && inputs <= 2 && p->mode != DFGPU_PW_GEN_INDEX) {
        int order[DFGPU_MAX_RANK], count = 0;
        DenseOperand a{}, b{};
        if (dense_order(p->out, order, count) && dense_operand(p->in0, p->out, order, count, tensors[0], a) &&
            dense_operand(binary ? p->in1 : p->in0, p->out, order, count, binary ? tensors[1] : tensors[0], b)) {
            if (f32_all) launch_dense<float>(inputs, a, b, tensors[2], p->mode, s, total, stream);
            else if (f16_all) launch_dense<__half>(inputs, a, b, tensors[2], p->mode, s, total, stream);
            else launch_dense<__nv_bfloat16>(inputs, a, b, tensors[2], p->mode, s, total, stream);
            return check_launch("POINTWISE");
        }
    }
    if (!simple_mode(p->mode)) {
        unsigned grid = static_cast<unsigned>((total + 255) / 256);
        launch_chained(pointwise_general_kernel, dim3(grid), dim3(256), 0, stream, tensors[0], tensors[1], inputs >= 3 ? tensors[3] : nullptr, tensors[2],
                                                           make_view(p->in0), inputs >= 2 ? make_view(p->in1) : make_view(p->in0),
                                                           inputs >= 3 ? make_view(p->in2) : make_view(p->in0), make_view(p->out),
                                                           p->mode, s, total);
    } else {
        unsigned grid = static_cast<unsigned>((total + 255) / 256);
        launch_chained(pointwise_kernel, dim3(grid), dim3(256), 0, stream, tensors[0], tensors[1], tensors[2], make_view(p->in0),
                                                   binary ? make_view(p->in1) : make_view(p->in0), make_view(p->out),
                                                   p->mode, p->relu_lower, p->relu_upper, p->relu_slope, total);
    }
    return check_launch("POINTWISE");
}
