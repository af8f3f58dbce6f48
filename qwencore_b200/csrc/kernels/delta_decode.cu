// Gated DeltaNet recurrent decode step on int8 state with a per-row fp32 scale.
//
// Replaces crates/qwc-cuda/cuda/delta_net.cu:1220-1237 (qwc_delta_decode_int8) behind the
// same C signature.  Arithmetic per state row (cuda/delta_net.cu:99-119,137-175):
//   s = float(code) * scale;  u = s.k;  w = s.q;  c = beta (v - alpha u)
//   s <- alpha s + c k;  out = alpha w + c (k.q)
//   peak = max|s|; inverse = 127 / peak; code = rint(s * inverse); scale = peak * (1/127)
//
// The op reads and rewrites 16 KiB + 512 B per (slot, value head) and nothing else of
// size, so it is bound by HBM read+write bandwidth.  Layout for sm_100a:
//   * one CTA per (value head, slot, row split); the state tile is brought into shared
//     memory by bulk-async copies (TMA 1-D) in 4 KiB quarters, each signalling its own
//     mbarrier, so the first rows are processed while the rest are in flight, and the
//     requantised tile leaves by one bulk store;
//   * the two dot products of a row run on the integer tensor cores: the codes are s8 already, and k
//     and q enter as four s8 digits each of a 31-bit fixed-point number (one binary exponent per
//     vector), so that one m16n8k32 instruction multiplies 16 rows by all eight digit columns.  The
//     sums are exact in s32 and are rounded once, when the digits are put together: closer to the
//     real product than the fp32 chain that rounds each of its 128 steps;
//   * the update: eight lanes share a row (16 codes each) when the grid is deep enough to keep seven CTAs
//     per SM resident - their warps hide the dependent-instruction latency that bounds the kernel
//     beside its issue slots - and four lanes (32 codes each) when all CTAs fit the SMs at four each
//     (kernel_for);
//   * the elementwise fp32 work uses the packed f32x2 pipe, and both int8 <-> fp32
//     conversions are bit tricks on the 2^23 binade (exact, round-to-nearest-even),
//     which keeps the instruction count under what the memory stream allows.
//
// The requantiser rounds exactly as the reference's: multiply by `127 / peak` in fp32,
// round to nearest even, scale = peak * (1/127); a zero row stores codes 0 and scale 0.

#include "common.cuh"

namespace qwc {
namespace {

constexpr int kDim = kDeltaHeadDim;  // 128 x 128 state per head
constexpr int kThreads = 128;
constexpr int kPartRows = 32;        // rows per bulk copy / per CTA iteration
constexpr int kMaxParts = kDim / kPartRows;

__device__ __forceinline__ float2 f2(float a, float b) { return make_float2(a, b); }

// D[16 rows][8] += A[16][32] (s8, row major) x B[32][8] (s8, column major), exact in s32.
__device__ __forceinline__ void mma_s8_16832(int (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// Fixed point is for vectors whose largest magnitude lies in [2^-90, 2^91) (or that are all zero);
// anything else - infinities and NaN among it - takes the fp32 sums of dots_fp32.
constexpr uint32_t kFixedLowest = 37u << 23;
constexpr uint32_t kFixedBeyond = 218u << 23;

__device__ __forceinline__ bool fixed_point_fits(uint32_t peak_bits) {
    return peak_bits == 0u || (peak_bits >= kFixedLowest && peak_bits < kFixedBeyond);
}

// x as a multiple of 2^(E - 30), E the exponent with peak < 2^E, in four balanced s8 digits (byte j
// counts 256^j).
__device__ __forceinline__ uint32_t fixed_digits(float x, uint32_t peak_bits) {
    const float up = peak_bits == 0u ? 0.0f : __uint_as_float((283u - (peak_bits >> 23)) << 23);
    return (static_cast<uint32_t>(__float2int_rn(x * up)) + 0x00808080u) ^ 0x00808080u;
}

__device__ __forceinline__ float fixed_unit(uint32_t peak_bits) {
    return peak_bits == 0u ? 0.0f : __uint_as_float(((peak_bits >> 23) - 29u) << 23);
}

// Row . k and row . q in fp32 for vectors outside the fixed-point range: four lanes per row.
__device__ __noinline__ float2 dots_fp32(const uint8_t* row, float scale, const float* k, const float* q, int t) {
    float u = 0.0f, w = 0.0f;
#pragma unroll 1
    for (int i = t; i < kDim; i += 4) {
        const float s = static_cast<float>(static_cast<int8_t>(row[i])) * scale;
        u = fmaf(s, k[i], u);
        w = fmaf(s, q[i], w);
    }
#pragma unroll
    for (int offset = 1; offset < 4; offset <<= 1) {
        u += __shfl_xor_sync(0xffffffffu, u, offset);
        w += __shfl_xor_sync(0xffffffffu, w, offset);
    }
    return make_float2(u, w);
}

__device__ __forceinline__ float max3_magnitude(float2 s, float peak) {
    return fmaxf(fmaxf(fabsf(s.x), fabsf(s.y)), peak);
}

// What the fused output stage needs (the gated RMSNorm of cuda/delta_output.cu:20-64 on this CTA's head,
// staged for the output projection); `staged == nullptr`: no fusion, `out` is written instead.
struct GatedNorm {
    const __nv_bfloat16* weight;  // [128]
    const float* gate_sums;       // the in-projection's K-split slices [slices][batch][width], or null
    const __nv_bfloat16* gate_rows;  // ... or its bf16 rows with `gate_stride` elements per row
    int slices;
    int batch;
    int width;
    int gate_column;  // of z within a row
    float gate_scale;
    float epsilon;
    __half* staged;   // [heads * 128 / 8][padded rows][8]
    int padded_rows;
};

// `kEarly`: the rows' state slots were fixed when the step was packed and a layer's state is written by
// nobody but this kernel, so the slot lookup and the copies of the state tile are issued before the
// wait for the preceding kernel (which produces q, k, v and the gates).  Callers outside a step, who
// may have written slots or state just before on the same stream, get the conservative order.
//
// `kLanes`: lanes that share a row in the update.  Eight: 16 elements each, 66 registers, seven CTAs per
// SM.  Four: 32 elements each, 105 registers, four CTAs per SM, but a third fewer instructions and half
// as many dependent steps per warp (see kernel_for).
template <bool kEarly, int kLanes>
__global__ void __launch_bounds__(kThreads, kLanes == 8 ? 7 : 4) delta_decode_int8_kernel(
    int8_t* __restrict__ state, float* __restrict__ state_scales, const uint32_t* __restrict__ state_slots,
    const float* __restrict__ q, const float* __restrict__ k, const float* __restrict__ v,
    const float* __restrict__ alpha, const float* __restrict__ beta, const float* __restrict__ kq,
    float* __restrict__ out, int v_heads, int state_capacity, int* status, const GatedNorm norm) {
    pdl_launch_dependents();
    __shared__ __align__(128) uint8_t tile[kDim * kDim];
    __shared__ __align__(16) float row_scale[kDim];
    __shared__ float out_rows[kDim];
    __shared__ float change_rows[kDim];  // eight lanes: c of every row
    __shared__ __align__(16) float v_rows[kDim];
    __shared__ __align__(16) uint32_t digits[2][kDim];  // k and q in fixed point
    __shared__ uint32_t peaks[2][kThreads / 32];
    __shared__ uint32_t b_words[kLanes == 8 ? 1 : 8][32];  // B fragments: [word of the lane's codes][lane]
    __shared__ uint64_t bars[kMaxParts];
    __shared__ int failed;

    const int rows_here = kDim / gridDim.z;
    const int parts = (rows_here + kPartRows - 1) / kPartRows;
    const int part_rows = rows_here < kPartRows ? rows_here : kPartRows;
    if (threadIdx.x == 0) {
        failed = 0;
        for (int part = 0; part < parts; ++part) {
            mbar_init(&bars[part], 1);
        }
        mbar_fence_init();
    }
    if (!kEarly) {
        pdl_wait();
    }
    const int h = blockIdx.x;
    const int b = blockIdx.y;
    const int row_begin = blockIdx.z * rows_here;
    const int slot = state_slots == nullptr ? b : static_cast<int>(state_slots[b]);
    if (status_is_set(status)) {  // (after the slot was asked for: one round trip for both)
        return;
    }
    if (static_cast<uint32_t>(slot) >= static_cast<uint32_t>(state_capacity)) {
        // a slot beyond the pool: nothing of this row is read or written, the host learns of it
        // through the status word (the whole CTA takes this branch: the slot is per row)
        if (threadIdx.x == 0) {
            atomicCAS(status, 0, kStatusStateSlotRange);
        }
        return;
    }
    const int hk = h / (v_heads / kDeltaKeyHeads);

    int8_t* S = state + (static_cast<size_t>(slot) * v_heads + h) * (kDim * kDim) + row_begin * kDim;
    float* scales = state_scales + (static_cast<size_t>(slot) * v_heads + h) * kDim + row_begin;

    // the thread that set the barriers up is the one that uses them here
    if (threadIdx.x == 0) {
        for (int part = 0; part < parts; ++part) {
            const uint32_t bytes = part_rows * kDim;
            mbar_arrive_expect_tx(&bars[part], bytes + (part == 0 ? rows_here * 4 : 0));
            bulk_g2s(tile + part * kPartRows * kDim, S + part * kPartRows * kDim, bytes, &bars[part]);
            if (part == 0) {
                bulk_g2s(row_scale, scales, rows_here * 4, &bars[0]);
            }
        }
    }
    if (kEarly) {
        pdl_wait();  // q, k, v and the gates come from the preceding kernel
    }
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const float* k_head = k + (static_cast<size_t>(b) * kDeltaKeyHeads + hk) * kDim;
    const float* q_head = q + (static_cast<size_t>(b) * kDeltaKeyHeads + hk) * kDim;
    const float my_k = k_head[threadIdx.x];  // a thread per element of the key head
    const float my_q = q_head[threadIdx.x];
    const int g = lane >> 2;  // row of an eight
    const int t = lane & 3;   // the lane's columns of the row: 16 t .. + 15 and 64 + 16 t .. + 15
    // eight lanes: the lane's columns in the update are 16 sub .. + 15
    const int sub = lane & 7;
    const int row_in_warp = lane >> 3;
    float2 kk[64 / kLanes];
#pragma unroll
    for (int i = 0; i < 32 / kLanes; ++i) {
        const int column = kLanes == 8 ? 16 * sub + 4 * i : 64 * (i >> 2) + 16 * t + 4 * (i & 3);
        const float4 kv = *reinterpret_cast<const float4*>(k_head + column);
        kk[2 * i] = f2(kv.x, kv.y);
        kk[2 * i + 1] = f2(kv.z, kv.w);
    }
    if (threadIdx.x < rows_here) {
        v_rows[threadIdx.x] = v[(static_cast<size_t>(b) * v_heads + h) * kDim + row_begin + threadIdx.x];
    }
    const float a = alpha[static_cast<size_t>(b) * v_heads + h];
    const float bt = beta[static_cast<size_t>(b) * v_heads + h];
    const float kq_token = kq[static_cast<size_t>(b) * kDeltaKeyHeads + hk];

    const uint32_t k_peak_warp = __reduce_max_sync(0xffffffffu, __float_as_uint(my_k) & 0x7fffffffu);
    const uint32_t q_peak_warp = __reduce_max_sync(0xffffffffu, __float_as_uint(my_q) & 0x7fffffffu);
    if (lane == 0) {
        peaks[0][warp] = k_peak_warp;
        peaks[1][warp] = q_peak_warp;
    }
    __syncthreads();
    uint32_t k_peak = 0, q_peak = 0;  // the largest magnitudes as bits: ordered like the magnitudes, NaN above all
#pragma unroll
    for (int i = 0; i < kThreads / 32; ++i) {
        k_peak = max(k_peak, peaks[0][i]);
        q_peak = max(q_peak, peaks[1][i]);
    }
    const bool fixed = fixed_point_fits(k_peak) && fixed_point_fits(q_peak);
    if (fixed) {
        digits[0][threadIdx.x] = fixed_digits(my_k, k_peak);
        digits[1][threadIdx.x] = fixed_digits(my_q, q_peak);
    }
    __syncthreads();

    // B fragments: column g is digit g & 3 of k (g < 4) or q.  The contraction is over columns in the
    // order in which a lane holds its codes: chunk c of lane t is columns 16 (4 c + t) .. + 15.
    // Eight lanes: every warp gathers all of them for itself.  Four lanes have no registers to keep them
    // in: a warp gathers a quarter of them for all.
    uint32_t b_own[8];
    {
        const uint32_t pick = (g & 3) | ((4 + (g & 3)) << 4);
        const auto gather = [&](int word) {
            const uint4 four =
                *reinterpret_cast<const uint4*>(digits[g >> 2] + 16 * (4 * (word >> 2) + t) + 4 * (word & 3));
            return __byte_perm(__byte_perm(four.x, four.y, pick), __byte_perm(four.z, four.w, pick), 0x5410);
        };
        if constexpr (kLanes == 8) {
#pragma unroll
            for (int word = 0; word < 8; ++word) {
                b_own[word] = gather(word);
            }
        } else {
            b_words[2 * warp][lane] = gather(2 * warp);
            b_words[2 * warp + 1][lane] = gather(2 * warp + 1);
            __syncthreads();
        }
    }
    const auto b_word = [&](int word) { return kLanes == 8 ? b_own[word] : b_words[word][lane]; };
    const float unit = fixed_unit(t < 2 ? k_peak : q_peak) * ((t & 1) ? 65536.0f : 1.0f);

    constexpr float kMagic = 12582912.0f;        // 1.5 * 2^23
    constexpr float kMagicBiased = 12583040.0f;  // kMagic + 128

    // A warp takes 16 rows at a time: rows 16 warp .. of the first 64, then of the last 64.
    for (int first = 16 * warp; first < rows_here; first += 16 * (kThreads / 32)) {
        // a warp leaves as a whole: the row reductions below are full-warp shuffles
        const bool arrived = __all_sync(
            0xffffffffu, mbar_wait_bounded(&bars[first / kPartRows], 0, kStatusDeltaTileWait, status) &&
                             (first < kPartRows || mbar_wait_bounded(&bars[0], 0, kStatusDeltaTileWait, status)));
        if (!arrived) {
            failed = 1;
            break;
        }
        // rows g and g + 8 of the sixteen; the second eight are absent when the split leaves eight rows
        const int row_lo = first + g;
        const int row_hi = min(first + g + 8, rows_here - 1);
        float u[2], w[2];
        if (fixed) {
            int sums[4] = {0, 0, 0, 0};
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                const uint4 lo = *reinterpret_cast<const uint4*>(tile + row_lo * kDim + 16 * (4 * c + t));
                const uint4 hi = *reinterpret_cast<const uint4*>(tile + row_hi * kDim + 16 * (4 * c + t));
                const uint32_t a0[4] = {lo.x, hi.x, lo.y, hi.y};
                const uint32_t a1[4] = {lo.z, hi.z, lo.w, hi.w};
                mma_s8_16832(sums, a0, b_word(4 * c), b_word(4 * c + 1));
                mma_s8_16832(sums, a1, b_word(4 * c + 2), b_word(4 * c + 3));
            }
            // this lane: two digits of k (t < 2) or q, the low two (t even) or the high two
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const float part =
                    fmaf(static_cast<float>(sums[2 * r + 1]), 256.0f, static_cast<float>(sums[2 * r])) * unit;
                const float whole = part + __shfl_xor_sync(0xffffffffu, part, 1);
                const float other = __shfl_xor_sync(0xffffffffu, whole, 2);
                u[r] = t < 2 ? whole : other;
                w[r] = t < 2 ? other : whole;
            }
        } else {
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const int row = r == 0 ? row_lo : row_hi;
                const float2 both = dots_fp32(tile + row * kDim, row_scale[row], k_head, q_head, t);
                u[r] = both.x;
                w[r] = both.y;
            }
        }
        if constexpr (kLanes == 8) {
            if (t < 2) {  // lane t finishes row g (t = 0) or g + 8
                const int row = t == 0 ? row_lo : row_hi;
                const float scale = row_scale[row];
                // (an infinite scale marks a row that has overflowed: its dots are NaN, as 0 * inf is)
                const float dot_k = fmaf(t == 0 ? u[0] : u[1], fixed ? scale : 1.0f, scale - scale);
                const float dot_q = fmaf(t == 0 ? w[0] : w[1], fixed ? scale : 1.0f, scale - scale);
                const float c = bt * (v_rows[row] - a * dot_k);
                change_rows[row] = c;
                out_rows[row] = a * dot_q + c * kq_token;
            }
            __syncwarp();

#pragma unroll 1
            for (int pass = 0; pass < 4; ++pass) {
                if (first + pass * 4 >= rows_here) {
                    break;
                }
                const int local = first + pass * 4 + row_in_warp;
                uint8_t* row_ptr = tile + local * kDim + 16 * sub;
                const uint4 codes = *reinterpret_cast<const uint4*>(row_ptr);
                const float scale = row_scale[local];
                const float c = change_rows[local];

                const uint32_t words[4] = {codes.x, codes.y, codes.z, codes.w};
                float2 s[8];
                const float2 bias = f2(-kMagicBiased, -kMagicBiased);
                const float2 scale2 = f2(scale, scale);
                const float2 a2 = f2(a, a);
                const float2 cc = f2(c, c);
                float peak = 0.0f;
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const uint32_t x = words[i] ^ 0x80808080u;
                    const float2 lo = f2(__uint_as_float(__byte_perm(x, 0x4B400000u, 0x7650)),
                                         __uint_as_float(__byte_perm(x, 0x4B400000u, 0x7651)));
                    const float2 hi = f2(__uint_as_float(__byte_perm(x, 0x4B400000u, 0x7652)),
                                         __uint_as_float(__byte_perm(x, 0x4B400000u, 0x7653)));
                    s[2 * i] = __ffma2_rn(cc, kk[2 * i], __fmul2_rn(a2, __fmul2_rn(__fadd2_rn(lo, bias), scale2)));
                    s[2 * i + 1] = __ffma2_rn(cc, kk[2 * i + 1], __fmul2_rn(a2, __fmul2_rn(__fadd2_rn(hi, bias), scale2)));
                    peak = max3_magnitude(s[2 * i], peak);
                    peak = max3_magnitude(s[2 * i + 1], peak);
                }
#pragma unroll
                for (int offset = 1; offset < 8; offset <<= 1) {
                    peak = fmaxf(peak, __shfl_xor_sync(0xffffffffu, peak, offset));
                }

                const float inverse = peak == 0.0f ? 0.0f : __fdiv_rn(127.0f, peak);
                const float2 inverse2 = f2(inverse, inverse);
                const float2 magic2 = f2(kMagic, kMagic);
                uint32_t packed[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float2 y0 = __fadd2_rn(__fmul2_rn(s[2 * i], inverse2), magic2);
                    const float2 y1 = __fadd2_rn(__fmul2_rn(s[2 * i + 1], inverse2), magic2);
                    const uint32_t lo = __byte_perm(__float_as_uint(y0.x), __float_as_uint(y0.y), 0x0040);
                    const uint32_t hi = __byte_perm(__float_as_uint(y1.x), __float_as_uint(y1.y), 0x0040);
                    packed[i] = __byte_perm(lo, hi, 0x5410);
                }
                *reinterpret_cast<uint4*>(row_ptr) = make_uint4(packed[0], packed[1], packed[2], packed[3]);
                if (sub == 0) {
                    row_scale[local] = __fmul_rn(peak, 1.0f / 127.0f);
                }
            }
        } else {
#pragma unroll 1
            for (int r = 0; r < 2; ++r) {
                const int local = r == 0 ? row_lo : row_hi;
                const float scale = row_scale[local];
                // (an infinite scale marks a row that has overflowed: its dots are NaN, as 0 * inf is)
                const float dot_k = fmaf(r == 0 ? u[0] : u[1], fixed ? scale : 1.0f, scale - scale);
                const float dot_q = fmaf(r == 0 ? w[0] : w[1], fixed ? scale : 1.0f, scale - scale);
                const float c = bt * (v_rows[local] - a * dot_k);
                const float contribution = a * dot_q + c * kq_token;
                uint8_t* const at = tile + local * kDim + 16 * t;
                const uint4 first_codes = *reinterpret_cast<const uint4*>(at);
                const uint4 second_codes = *reinterpret_cast<const uint4*>(at + 64);
                const uint32_t words[8] = {first_codes.x,  first_codes.y,  first_codes.z,  first_codes.w,
                                           second_codes.x, second_codes.y, second_codes.z, second_codes.w};
                float2 s[16];
                const float2 bias = f2(-kMagicBiased, -kMagicBiased);
                const float2 scale2 = f2(scale, scale);
                const float2 a2 = f2(a, a);
                const float2 cc = f2(c, c);
                float peak_a = 0.0f, peak_b = 0.0f;
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const uint32_t x = words[i] ^ 0x80808080u;
                    const float2 lo = f2(__uint_as_float(__byte_perm(x, 0x4B400000u, 0x7650)),
                                         __uint_as_float(__byte_perm(x, 0x4B400000u, 0x7651)));
                    const float2 hi = f2(__uint_as_float(__byte_perm(x, 0x4B400000u, 0x7652)),
                                         __uint_as_float(__byte_perm(x, 0x4B400000u, 0x7653)));
                    s[2 * i] = __ffma2_rn(cc, kk[2 * i], __fmul2_rn(a2, __fmul2_rn(__fadd2_rn(lo, bias), scale2)));
                    s[2 * i + 1] = __ffma2_rn(cc, kk[2 * i + 1], __fmul2_rn(a2, __fmul2_rn(__fadd2_rn(hi, bias), scale2)));
                    peak_a = max3_magnitude(s[2 * i], peak_a);
                    peak_b = max3_magnitude(s[2 * i + 1], peak_b);
                }
                float peak = fmaxf(peak_a, peak_b);
#pragma unroll
                for (int offset = 1; offset < 4; offset <<= 1) {
                    peak = fmaxf(peak, __shfl_xor_sync(0xffffffffu, peak, offset));
                }

                const float inverse = peak == 0.0f ? 0.0f : __fdiv_rn(127.0f, peak);
                const float2 inverse2 = f2(inverse, inverse);
                const float2 magic2 = f2(kMagic, kMagic);
                uint32_t packed[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const float2 y0 = __fadd2_rn(__fmul2_rn(s[2 * i], inverse2), magic2);
                    const float2 y1 = __fadd2_rn(__fmul2_rn(s[2 * i + 1], inverse2), magic2);
                    const uint32_t lo = __byte_perm(__float_as_uint(y0.x), __float_as_uint(y0.y), 0x0040);
                    const uint32_t hi = __byte_perm(__float_as_uint(y1.x), __float_as_uint(y1.y), 0x0040);
                    packed[i] = __byte_perm(lo, hi, 0x5410);
                }
                if (first + g + 8 * r < rows_here) {
                    *reinterpret_cast<uint4*>(at) = make_uint4(packed[0], packed[1], packed[2], packed[3]);
                    *reinterpret_cast<uint4*>(at + 64) = make_uint4(packed[4], packed[5], packed[6], packed[7]);
                    if (t == 0) {
                        row_scale[local] = __fmul_rn(peak, 1.0f / 127.0f);
                        out_rows[local] = contribution;
                    }
                }
            }
        }
    }

    fence_proxy_async();
    __syncthreads();
    if (failed) {
        // The copies that were asked for may still be landing in this CTA's shared memory: their
        // thread waits for each of them (bounded) before the CTA gives the memory back.
        if (threadIdx.x == 0) {
            for (int part = 0; part < parts; ++part) {
                mbar_wait_bounded(&bars[part], 0, kStatusDeltaTileWait, status);
            }
        }
        return;
    }
    if (threadIdx.x == 0) {
        bulk_s2g(S, tile, rows_here * kDim);
        bulk_s2g(scales, row_scale, rows_here * 4);
        bulk_commit();
    }
    if (norm.staged != nullptr) {
        // The whole head is here (the launcher fuses only unsplit heads): gated RMSNorm and the staged
        // store, thread = dimension.  Rounding points as cuda/delta_output.cu:38-64.
        __shared__ float warp_sums[kThreads / 32];
        const int dimension = threadIdx.x;
        const int column = norm.gate_column + h * kDim + dimension;
        float gate_value;
        if (norm.gate_sums != nullptr) {
            const size_t stride = static_cast<size_t>(norm.batch) * norm.width;
            const float* at = norm.gate_sums + static_cast<size_t>(b) * norm.width + column;
            float total = 0.0f;
            for (int first = 0; first < norm.slices; first += 4) {
                float part[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    part[j] = __ldcg(at + min(first + j, norm.slices - 1) * stride);
                }
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    total += first + j < norm.slices ? part[j] : 0.0f;
                }
            }
            gate_value = __bfloat162float(__float2bfloat16(total * norm.gate_scale));
        } else {
            gate_value = __bfloat162float(norm.gate_rows[static_cast<size_t>(b) * norm.width + column]);
        }
        const float gain = __bfloat162float(norm.weight[dimension]);
        const float value = __bfloat162float(__float2bfloat16(out_rows[dimension]));
        float sum = warp_sum(value * value);
        if ((threadIdx.x & 31) == 0) {
            warp_sums[threadIdx.x >> 5] = sum;
        }
        __syncthreads();
        sum = 0.0f;
        for (int w = 0; w < kThreads / 32; ++w) {
            sum += warp_sums[w];
        }
        const float inverse = rsqrtf(sum / static_cast<float>(kDim) + norm.epsilon);
        const __nv_bfloat16 normalized = __float2bfloat16(value * inverse);
        const __nv_bfloat16 weighted = __float2bfloat16(gain * __bfloat162float(normalized));
        const float silu = gate_value / (1.0f + __expf(-gate_value));
        const __nv_bfloat16 result = __float2bfloat16(__bfloat162float(weighted) * silu);
        const int feature = h * kDim + dimension;
        norm.staged[(static_cast<size_t>(feature >> 3) * norm.padded_rows + b) * 8 + (feature & 7)] =
            __float2half_rn(fminf(fmaxf(__bfloat162float(result), -65504.0f), 65504.0f));
    } else {
        float* op = out + (static_cast<size_t>(b) * v_heads + h) * kDim + row_begin;
        for (int i = threadIdx.x; i < rows_here; i += kThreads) {
            op[i] = out_rows[i];
        }
    }
    if (threadIdx.x == 0) {
        bulk_wait_all_read();
    }
}

int sm_count_delta() {
    int device = 0, value = 0;
    if (cudaGetDevice(&device) == cudaSuccess &&
        cudaDeviceGetAttribute(&value, cudaDevAttrMultiProcessorCount, device) == cudaSuccess && value > 0) {
        return value;
    }
    return 148;
}

// Row splits so that the grid has at least two CTAs per SM
// (same purpose as splits_for, cuda/delta_net.cu:1184-1200).
int splits_for(int batch, int v_heads) {
    const int sms = sm_count_delta();
    const int base = v_heads * batch;
    int split = 1;
    while (split < 8 && base * split < 2 * sms) {
        split *= 2;
    }
    return split;
}

using DeltaKernel = void (*)(int8_t*, float*, const uint32_t*, const float*, const float*, const float*, const float*,
                             const float*, const float*, float*, int, int, int*, const GatedNorm);

// Four lanes per row while every CTA is resident at once with them (four per SM), eight beyond.
// Measured (us, layers that L2 does not hold, four / eight lanes): 48 heads at 1 row 3.54 / 4.62, at 9
// rows (432 CTAs) 7.7 / 11.1; 32 heads at 32 rows (1024 CTAs, two waves of the first) 13.6 / 12.5.
// (The fp32 dot products that the integer tensor cores replaced: 4.94, 12.06 and 14.0.)
template <bool kEarly>
DeltaKernel kernel_for(int ctas) {
    return ctas <= 4 * sm_count_delta() ? delta_decode_int8_kernel<kEarly, 4> : delta_decode_int8_kernel<kEarly, 8>;
}

}  // namespace
}  // namespace qwc

extern "C" int qwc_delta_decode_int8(void* state, float* state_scales, const void* state_slots, const void* q,
                                     const void* k, const void* v, const void* alpha, const void* beta,
                                     const void* kq, void* out, int state_capacity, int batch,
                                     cudaStream_t stream) {
    if (state == nullptr || state_scales == nullptr || q == nullptr || k == nullptr || v == nullptr ||
        alpha == nullptr || beta == nullptr || kq == nullptr || out == nullptr || state_capacity < batch ||
        batch <= 0 || batch > qwc::kMaxDecodeBatch) {
        return cudaErrorInvalidValue;
    }
    const int v_heads = qwc::current_shape().delta_value_heads;
    int* status = qwc::status_ptr();
    if (status == nullptr) {
        return cudaErrorInvalidValue;
    }
    const dim3 grid(v_heads, batch, qwc::splits_for(batch, v_heads));
    return qwc::launch_chained(qwc::kernel_for<false>(grid.x * grid.y * grid.z), dim3(grid), dim3(qwc::kThreads), 0, stream,
        static_cast<int8_t*>(state), state_scales, static_cast<const uint32_t*>(state_slots),
        static_cast<const float*>(q), static_cast<const float*>(k), static_cast<const float*>(v),
        static_cast<const float*>(alpha), static_cast<const float*>(beta), static_cast<const float*>(kq),
        static_cast<float*>(out), v_heads, state_capacity, status, qwc::GatedNorm{});
}

// The step's form of the same update (additive; the decode executor's own): the state slots and the
// state tiles are fetched while the preceding kernel still runs (see kEarly above), and when every head
// is one CTA (qwc_delta_decode_fuses_norm) the gated RMSNorm of qwc_delta_gated_rmsnorm_split /
// _staged runs in the same CTA and the result is stored staged for the output projection; `out` is
// then not written.  gate: either the in-projection's K-split slices (gate_sums, slices, scale) or its
// bf16 rows (gate_rows), `width` elements per row, z at column `gate_column`.
extern "C" int qwc_delta_decode_fuses_norm(int batch) {
    const int v_heads = qwc::current_shape().delta_value_heads;
    return batch > 0 && batch <= 32 && qwc::splits_for(batch, v_heads) == 1 ? 1 : 0;
}

extern "C" int qwc_delta_decode_int8_step(void* state, float* state_scales, const void* state_slots, const void* q,
                                          const void* k, const void* v, const void* alpha, const void* beta,
                                          const void* kq, void* out, int state_capacity, int batch,
                                          const float* gate_sums, int slices, float gate_global_scale,
                                          const void* gate_rows, int width, int gate_column,
                                          const void* norm_weight, float epsilon, void* staged_output,
                                          cudaStream_t stream) {
    if (state == nullptr || state_scales == nullptr || state_slots == nullptr || q == nullptr || k == nullptr ||
        v == nullptr || alpha == nullptr || beta == nullptr || kq == nullptr || out == nullptr ||
        state_capacity < batch || batch <= 0 || batch > qwc::kMaxDecodeBatch) {
        return cudaErrorInvalidValue;
    }
    const int v_heads = qwc::current_shape().delta_value_heads;
    int* status = qwc::status_ptr();
    if (status == nullptr) {
        return cudaErrorInvalidValue;
    }
    const int splits = qwc::splits_for(batch, v_heads);
    qwc::GatedNorm norm = {};
    if (staged_output != nullptr) {
        if (splits != 1 || batch > 32 || norm_weight == nullptr || (gate_sums == nullptr && gate_rows == nullptr) ||
            (gate_sums != nullptr && (slices <= 0 || slices > 64 || !(gate_global_scale > 0.0f))) ||
            gate_column < 0 || gate_column + v_heads * qwc::kDim > width || !isfinite(epsilon) || epsilon <= 0.0f) {
            return cudaErrorInvalidValue;
        }
        norm.weight = static_cast<const __nv_bfloat16*>(norm_weight);
        norm.gate_sums = gate_sums;
        norm.gate_rows = static_cast<const __nv_bfloat16*>(gate_rows);
        norm.slices = slices;
        norm.batch = batch;
        norm.width = width;
        norm.gate_column = gate_column;
        norm.gate_scale = gate_sums != nullptr ? 1.0f / gate_global_scale : 1.0f;
        norm.epsilon = epsilon;
        norm.staged = static_cast<__half*>(staged_output);
        norm.padded_rows = batch <= 16 ? 16 : 32;
    }
    const dim3 grid(v_heads, batch, splits);
    return qwc::launch_chained(qwc::kernel_for<true>(grid.x * grid.y * grid.z), dim3(grid), dim3(qwc::kThreads), 0, stream,
        static_cast<int8_t*>(state), state_scales, static_cast<const uint32_t*>(state_slots),
        static_cast<const float*>(q), static_cast<const float*>(k), static_cast<const float*>(v),
        static_cast<const float*>(alpha), static_cast<const float*>(beta), static_cast<const float*>(kq),
        static_cast<float*>(out), v_heads, state_capacity, status, norm);
}
