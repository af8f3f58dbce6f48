// Packed-GQA paged attention over an e4m3 KV cache for ragged decode rows.
//
// Replaces crates/qwc-cuda/cuda/paged_attention.cu:1913-1958 (qwc_paged_attention_packed_fp8)
// for decode rows (tile of six packed query heads per KV head).  Semantics follow the
// reference: softmax and accumulation in fp32, optional sigmoid output gate, split-context partials
// merged by a second kernel (cuda/paged_attention.cu:1464-1574,1736-1823).
//
// The op reads every K and V byte of the row's context once and nothing else of
// size, so it is HBM-bound.  Layout for sm_100a:
//   * one CTA per SM at a time.  The rows of a ragged batch differ in context by orders of magnitude, so the
//     work is cut on the device (attention_plan.h): the 16-token units of all (row, kv head) pairs are laid end
//     to end, chunks of that line are dealt to the CTAs, and a task is the piece of one pair inside one chunk (its
//     partial is merged by the second kernel).  Up to 192 units per SM a chunk is an equal share of the line.
//     Beyond, there are a large chunk per SM and small ones, which go to whoever is done first: the grid has a
//     CTA for each, and a running CTA takes over those that have not started.  The launch shape depends on the SM
//     count, the rows and what the block tables could describe, not on the contexts, so the step stays
//     capturable in a CUDA graph;
//   * nobody converts a cache byte.  K and V go from memory to tcgen05.mma.kind::f8f6f4 as they are
//     stored: a stage is 128 tokens of one kv head, each unit of 16 tokens (a whole 16-token page, or a quarter
//     of a 64-token page) two swizzled TMA boxes of 128 bytes per token.  K is the A operand of S^T = K Q^T
//     (128 tokens x 256 dims, K-major), V the A operand of O^T = V^T P^T (dims x tokens, MN-major);
//   * queries and probabilities enter as e4m3 digits.  An e4m3 has four significant bits, so a number is written as
//     a sum of digits with powers of two for weights, every digit rounded to nearest from what the digits before it
//     left, and digit j of head h is column 8 j + h of the B operand: one accumulator per digit and output, added
//     with their weights in fp32.  A head's query is first brought to [128, 256) by a power of two and takes four
//     digits, of weight 1, 2^-4, 2^-18 and 2^-23: the first two hold a bf16's eight bits down to 2^-14 of the
//     largest element, the others (and the overlap) from there on, so that every element is exact down to 2^-32 of
//     the binade of the largest.  That is all that f16, which the kernel used to multiply with, holds exactly (2^-17
//     to 65504), whichever keys are zero.  A probability is p0 + p1 / 16 + p2 / 256, kept to 2^-13 of itself (f16:
//     2^-12), down to 2^-26 of the largest;
//   * O of one stage is read from tensor memory and added to fp32 registers, where a change of the running
//     maximum costs one multiplication.
//
//   warps 0-3   softmax: thread = token of the stage.  S from tensor memory, maximum over the 128 tokens,
//               exponentials, digits of P to shared memory
//   warps 4-11  thread = output dim: the accumulators of O, the result
//   warp 12     issues the MMAs: S of stage n + 1 before O of stage n
//   warps 13,14 fetch K and V into rings of three stages, ahead across task boundaries
//   warps 15,16 the query's digits, half of the heads each
//   warp 17     the tasks of one chunk after the other
//
// What it took to get there: widening every cache byte to f16 for mma.sync kept the conversion unit 76 % busy
// and the stage on dependent instructions.  Measured (us, layers that L2 does not hold, before / now):
// 32 rows in [128, 2048] 26.4 / 23.1, one row of 2048 12.3 / 10.3, three rows of 32768 45.3 / 42.5 (6.1 TB/s while it
// streams), 32 rows log-uniform to 32768 82.8 / 77.0, 20 rows from 8192 to 32768 134.1 / 121.4 (6.1 TB/s all in all).
// The new operands alone, on the old plan and merge, gave 26.4 / 25.5 and 82.9 / 82.6: what had been hidden behind
// the conversions was the plan, the merge and CTAs that ended early (SplitPlan, reduce_partitions_kernel).
//
// Cache memory must hold finite e4m3 codes in every allocated page (a zero-initialised
// pool, as the reference allocates it): positions past the context are masked by
// zero probabilities, not skipped.

#include <algorithm>
#include "attention_plan.h"
#include "tcgen05.cuh"

namespace qwc {
namespace {

constexpr int kSoftmaxWarps = 4;
constexpr int kOutputWarps = 8;
constexpr int kFirstOutputWarp = kSoftmaxWarps;
constexpr int kMmaWarp = kFirstOutputWarp + kOutputWarps;
constexpr int kKeyWarp = kMmaWarp + 1;
constexpr int kValueWarp = kMmaWarp + 2;
constexpr int kFirstQueryWarp = kMmaWarp + 3;
constexpr int kQueryWarps = 2;
constexpr int kPlanWarp = kFirstQueryWarp + kQueryWarps;
constexpr int kListReaders = kPlanWarp;  // every warp before it reads the task lists
constexpr int kThreads = (kPlanWarp + 1) * 32;
constexpr int kStageTokens = kStageUnits * kUnitTokens;
constexpr int kBoxBytes = kUnitTokens * 128;            // half the dims of a unit
constexpr int kHalfBytes = kStageUnits * kBoxBytes;     // ... of a stage
constexpr int kStageBytes = 2 * kHalfBytes;             // K or V of a stage
constexpr int kStages = 3;
constexpr int kQueryDigits = 4;                         // of weight 1, 2^-4, 2^-18, 2^-23
constexpr int kProbabilityDigits = 3;                   // of weight 1, 2^-4, 2^-8
constexpr int kColumns = 32;                            // digit j of head h is column 8 j + h; the rest is not used
constexpr int kQueryBytes = kColumns * kHeadDim;        // B operand of S, K-major core matrices
constexpr int kProbabilityBytes = kColumns * kStageTokens;  // B operand of O, MN-major core matrices
constexpr int kTmemColumns = 256;
constexpr int kScoreColumn = 0;                         // two buffers
constexpr int kOutputColumn = 2 * kColumns;             // two buffers of two halves of the dims
constexpr int kPartialFloats = 2;
constexpr size_t kPartialBytes = 2 * sizeof(float) + kHeadDim * sizeof(__half);  // 520
constexpr float kLog2e = 1.4426950408889634f;

struct Task {
    int row;
    int kv_head;
    int part;
    int last;  // no piece of the pair after this one
    int unit_begin;
    int units;
    int context;  // tokens of the row, cut at the block table's capacity
};

struct Smem {
    uint8_t k[kStages][kStageBytes];  // [half of the dims][token][128 bytes], 128-byte swizzle
    uint8_t v[kStages][kStageBytes];
    uint8_t p[2][kProbabilityBytes];  // [column / 16][token][16]
    uint8_t q[2][kQueryBytes];        // [dim / 16][column][16]
    uint64_t k_full[kStages], k_empty[kStages];
    uint64_t v_full[kStages], v_empty[kStages];
    uint64_t q_ready[2], q_free[2];   // of a task's query
    uint64_t s_ready[2], s_free[2];   // of a stage: scores in tensor memory
    uint64_t max_ready[2];            // the four warps' maxima
    uint64_t p_ready[2], p_free[2];   // probabilities in shared memory
    uint64_t o_ready[2], o_free[2];   // outputs in tensor memory
    uint64_t t_ready[2], t_free[2];   // of a task: sums and maxima
    float warp_max[2][kSoftmaxWarps][8];
    float rescale[4][8];              // what a stage multiplies the sums of the stages before it with
    float query_scale[2][8];
    float task_sum[2][kSoftmaxWarps][8];
    float task_max[2][8];
    uint64_t list_ready[2], list_free[2];  // of a chunk: its tasks
    uint64_t list_wanted;           // every copy of the newest chunk has been asked for
    uint64_t claim_ready;
    ulonglong2 claim;               // what the hardware answered
    unsigned long long first_unit[kPlanRows + 1];  // (as Positions) prefix sum of the rows' units (a row without context counts one)
    Task tasks[2][kMaxListTasks];
    int task_count[2];              // -1: there is nothing left
    uint32_t tmem_base;
    int failed;                     // a wait gave up
    int stages_asked;               // of K, so far: a wait that spans more than a stage goes on while this grows
};

static_assert(sizeof(Smem) + 1024 <= 232448, "shared memory of a CTA");
static_assert(kMaxListTasks * sizeof(Task) <= kProbabilityBytes, "the rehearsal's list");
static_assert(kPlanKvHeads == kKvHeads, "the plan's pairs");
static_assert(kGqaGroup % kQueryWarps == 0, "as many heads for each query warp");

// Gives up after 20 ms in which the CTA asked for nothing new.  (Some waits span a whole task or chunk: the queries of
// the task after the next, the next list.  At 40 to 100 GB/s an SM streams a gigabyte in 20 ms, so on contexts of
// millions of tokens such a wait is longer than that while everything goes on.)
// (out of line, as in the projection kernels: a wait that is already satisfied costs one test)
__device__ __noinline__ bool att_wait_slow(uint64_t* bar, uint32_t parity, Smem& sm, int* status) {
    long long start = clock64();
    int asked = *reinterpret_cast<volatile int*>(&sm.stages_asked);
    for (;;) {
#pragma unroll 1
        for (int spin = 0; spin < 64; ++spin) {
            if (mbar_try_wait(bar, parity)) {
                return true;
            }
        }
        if (*reinterpret_cast<volatile int*>(&sm.failed) != 0) {
            return false;
        }
        if (clock64() - start > 40000000ll) {
            const int asked_now = *reinterpret_cast<volatile int*>(&sm.stages_asked);
            if (asked_now == asked) {
                break;
            }
            asked = asked_now;
            start = clock64();
        }
    }
    atomicCAS(status, 0, kStatusAttentionPageWait);
    *reinterpret_cast<volatile int*>(&sm.failed) = 1;
    return false;
}

// For a converged warp: the same answer in every lane.
__device__ __forceinline__ bool att_wait(uint64_t* bar, uint32_t parity, Smem& sm, int* status) {
    const bool ok = mbar_try_wait(bar, parity) || att_wait_slow(bar, parity, sm, status);
    return __all_sync(0xffffffffu, ok);
}

// Operand of 128-byte rows with the 128-byte swizzle, eight rows (1 KiB) to an atom: K-major (a row is a token, its
// bytes the dims that are contracted) as well as MN-major (a row is a token that is contracted, its bytes the dims
// of the output).
__device__ __forceinline__ uint64_t swizzled_descriptor(uint32_t address) {
    const uint64_t lo = ((address >> 4) & 0x3FFFu) | (1ull << 16);
    const uint64_t hi = (1024u >> 4) | (1u << 14) | (2u << 29);
    return lo | (hi << 32);
}

// D[128][N] (+)= A[128][32] x B[N][32], e4m3 from shared memory, fp32 accumulate.
__device__ __forceinline__ void umma_fp8(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                         uint32_t accumulate) {
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "setp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], %1, %2, %3, p;\n"
        "}\n" ::"r"(d_tmem),
        "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}

__device__ __forceinline__ uint32_t float2_to_e4m3x2(float lo, float hi) {
    uint16_t out;
    asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;" : "=h"(out) : "f"(hi), "f"(lo));
    return out;
}

// The next digit of two numbers, and sixteen times what it leaves.
__device__ __forceinline__ uint32_t take_digit(float& lo, float& hi) {
    const uint32_t digit = float2_to_e4m3x2(lo, hi);
    const uint32_t half = cvt_e4m3x2_to_f16x2(digit);
    const float2 value = __half22float2(*reinterpret_cast<const __half2*>(&half));
    lo = (lo - value.x) * 16.0f;
    hi = (hi - value.y) * 16.0f;
    return digit;
}

__device__ __forceinline__ uint32_t f16x2_to_e4m3x2(__half2 value) {
    uint16_t out;
    asm("cvt.rn.satfinite.e4m3x2.f16x2 %0, %1;" : "=h"(out) : "r"(*reinterpret_cast<const uint32_t*>(&value)));
    return out;
}

__device__ __forceinline__ __half2 e4m3x2_to_half2(uint32_t digits) {
    const uint32_t value = cvt_e4m3x2_to_f16x2(digits);
    return *reinterpret_cast<const __half2*>(&value);
}

// The first two digits of two query elements, |x| < 256, in f16 arithmetic: exact, as all numbers in it have eight
// significant bits at most (an x below 2^-17 becomes a multiple of 2^-24, which costs nothing: the digits after these
// two start from x).  Together they are x itself from 2^-6 on, ...
__device__ __forceinline__ void take_high_digits(float lo, float hi, uint32_t& d0, uint32_t& d1) {
    const __half2 x = __floats2half2_rn(lo, hi);
    d0 = f16x2_to_e4m3x2(x);
    d1 = f16x2_to_e4m3x2(__hmul2(__hsub2(x, e4m3x2_to_half2(d0)), __float2half2_rn(16.0f)));
}

// ... and below they leave at most 2^-14 (a multiple of 2^-13 is what they make there), which the third holds as a
// normal number down to 2^-24 and the fourth finishes.
__device__ __forceinline__ void take_low_digits(float lo, float hi, uint32_t d0, uint32_t d1, uint32_t& d2, uint32_t& d3) {
    const float2 taken =
        __half22float2(__hfma2(e4m3x2_to_half2(d1), __float2half2_rn(0.0625f), e4m3x2_to_half2(d0)));
    const __half2 rest = __floats2half2_rn((lo - taken.x) * 262144.0f, (hi - taken.y) * 262144.0f);
    d2 = f16x2_to_e4m3x2(rest);
    d3 = f16x2_to_e4m3x2(__hmul2(__hsub2(rest, e4m3x2_to_half2(d2)), __float2half2_rn(32.0f)));
}

// Largest value of the warp (a NaN counts as nothing).
__device__ __forceinline__ float warp_highest(float value) {
    float out;
    asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(out) : "f"(value));
    return out;
}

// Asks the hardware for a CTA of this grid that has not started yet: it will not start, and whoever asked does its
// work.  The answer, 16 bytes, arrives in shared memory.
__device__ __forceinline__ void claim_chunk(ulonglong2* answer, uint64_t* bar) {
    asm volatile(
        "clusterlaunchcontrol.try_cancel.async.shared::cta.mbarrier::complete_tx::bytes.b128 [%0], [%1];" ::"r"(
            smem_u32(answer)),
        "r"(smem_u32(bar))
        : "memory");
}

// The CTA index in the answer, -1 when all have started (nothing may be asked after that).
__device__ __forceinline__ int claimed_chunk(const ulonglong2* answer) {
    int index;
    asm volatile(
        "{\n"
        ".reg .b128 answer;\n"
        ".reg .pred given;\n"
        ".reg .b32 x;\n"
        "ld.shared.b128 answer, [%1];\n"
        "clusterlaunchcontrol.query_cancel.is_canceled.pred.b128 given, answer;\n"
        "mov.b32 x, -1;\n"
        "@given clusterlaunchcontrol.query_cancel.get_first_ctaid::x.b32.b128 x, answer;\n"
        "mov.b32 %0, x;\n"
        "}\n"
        : "=r"(index)
        : "r"(smem_u32(answer))
        : "memory");
    return index;
}

// Accumulators of a digit each, with their weights: of probabilities ...
__device__ __forceinline__ float combine_digits(uint32_t d0, uint32_t d1, uint32_t d2) {
    return fmaf(fmaf(__uint_as_float(d2), 0.0625f, __uint_as_float(d1)), 0.0625f, __uint_as_float(d0));
}

// ... and of queries.
__device__ __forceinline__ float combine_query_digits(uint32_t d0, uint32_t d1, uint32_t d2, uint32_t d3) {
    const float low = fmaf(__uint_as_float(d3), 1.0f / 32.0f, __uint_as_float(d2));
    return fmaf(fmaf(low, 1.0f / 16384.0f, __uint_as_float(d1)), 0.0625f, __uint_as_float(d0));
}

// Cache pages as rows of 256 bytes, fetched in boxes of 16 tokens x 128 bytes.  The launcher does not know how many
// pages the pool has (nor do the kernels of the reference): the map describes as many rows as a coordinate can
// name, and the block tables say which of them exist.
cudaError_t encode_cache_map(CUtensorMap* map, const void* cache) {
    const EncodeTiled encode = tensor_map_encoder();
    if (encode == nullptr) {
        return cudaErrorNotSupported;
    }
    const cuuint64_t dims[2] = {kHeadDim, 0x7fffffffull};
    const cuuint64_t strides[1] = {kHeadDim};
    const cuuint32_t box[2] = {128, kUnitTokens};
    const cuuint32_t element_strides[2] = {1, 1};
    const CUresult result =
        encode(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(cache), dims, strides, box, element_strides,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return result == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

template <bool kSplit, typename Position>
__global__ void __launch_bounds__(kThreads, 1) paged_attention_packed_kernel(
    const __grid_constant__ CUtensorMap key_map, const __grid_constant__ CUtensorMap value_map,
    const __nv_bfloat16* __restrict__ query, const __nv_bfloat16* __restrict__ query_gate_projection,
    const uint32_t* __restrict__ block_tables, const uint32_t* __restrict__ context_lengths,
    const float* __restrict__ key_scales, const float* __restrict__ value_scales,
    __nv_bfloat16* __restrict__ output, __half* __restrict__ staged_output, int padded_rows,
    float* __restrict__ partial_stats, __half* __restrict__ partial_out, int rows, int max_blocks, int row_base,
    int page_size, int gate_stride, int partitions, int smallest_chunk, int ctas, float softmax_scale, int* status) {
    extern __shared__ unsigned char smem_raw[];
    Smem& sm = *reinterpret_cast<Smem*>(smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u));

    pdl_launch_dependents();
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const int units_per_page = page_size / kUnitTokens;
    const int capacity_units = max_blocks * units_per_page;

    if (warp == kMmaWarp) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sm.tmem_base)),
                     "r"(kTmemColumns)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    }
    if (threadIdx.x == kKeyWarp * 32) {
        for (int i = 0; i < kStages; ++i) {
            mbar_init(&sm.k_full[i], 1);
            mbar_init(&sm.k_empty[i], 1);
            mbar_init(&sm.v_full[i], 1);
            mbar_init(&sm.v_empty[i], 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&sm.q_ready[i], kQueryWarps);
            mbar_init(&sm.q_free[i], 1 + kSoftmaxWarps);
            mbar_init(&sm.s_ready[i], 1);
            mbar_init(&sm.s_free[i], kSoftmaxWarps);
            mbar_init(&sm.max_ready[i], kSoftmaxWarps);
            mbar_init(&sm.p_ready[i], kSoftmaxWarps);
            mbar_init(&sm.p_free[i], 1);
            mbar_init(&sm.o_ready[i], 2);  // the MMAs, and the thread that issued them (it passes on what it waited for)
            mbar_init(&sm.o_free[i], kOutputWarps);
            mbar_init(&sm.t_ready[i], kSoftmaxWarps);
            mbar_init(&sm.t_free[i], kOutputWarps);
            mbar_init(&sm.list_ready[i], 1);
            mbar_init(&sm.list_free[i], kListReaders);
        }
        mbar_init(&sm.list_wanted, 1);
        mbar_init(&sm.claim_ready, 1);
        sm.failed = 0;
        sm.stages_asked = 0;
        mbar_fence_init();
    }
    fence_proxy_async();
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(&sm.tmem_base);
    bool ok = true;
    int t = 0;  // tasks and ...
    int n = 0;  // ... stages so far, over all chunks
    int issued = 0;  // the MMA warp: O of this many stages
    int claims = 0;  // the plan warp: chunks asked for

    if (warp == kPlanWarp || warp == 0) {
        // ---------------- plan: the tasks of one chunk after the other ------------------------------
        // (Warp 0 walks through the first list too, into scratch, before the wait for the kernels ahead and on
        // whatever the context lengths are then: when the plan is made, its instructions are in the cache.)
        const bool rehearsal = warp == 0;
        if (!rehearsal) {
            pdl_wait();  // context lengths, tables, query and the cache rows of this step come from earlier kernels
        }
        Position* const first_unit =
            rehearsal ? reinterpret_cast<Position*>(sm.p[0]) : reinterpret_cast<Position*>(sm.first_unit);
        const int earlier_failure = *reinterpret_cast<const volatile int*>(status);
        SplitPlan<Position> plan = {};
        if (kSplit) {
            // prefix of the rows' units: a warp scan per 32 rows
            Position carry = 0;
#pragma unroll 1
            for (int base = 0; base < rows; base += 32) {
                const int r = base + lane;
                const Position mine =
                    r < rows ? plan_units(units_of_context(__ldcg(context_lengths + row_base + r), capacity_units)) : 0;
                Position inclusive = mine;
#pragma unroll
                for (int offset = 1; offset < 32; offset <<= 1) {
                    const Position other = __shfl_up_sync(0xffffffffu, inclusive, offset);
                    if (lane >= offset) {
                        inclusive += other;
                    }
                }
                if (r < rows) {
                    first_unit[r] = carry + inclusive - mine;
                }
                carry += __shfl_sync(0xffffffffu, inclusive, 31);
            }
            if (lane == 0) {
                first_unit[rows] = carry;
            }
            __syncwarp();
            plan = make_split_plan(carry, rows, smallest_chunk, ctas);
        }
        int chunk = earlier_failure != 0 ? -1 : static_cast<int>(blockIdx.x);
#pragma unroll 1
        for (int m = 0; ok; ++m) {
            Task* const tasks = rehearsal ? reinterpret_cast<Task*>(sm.p[1]) : sm.tasks[m & 1];
            int count = 0;
            if (chunk < 0) {
                count = -1;
            } else if (!kSplit) {
                // whole (row, kv head) pairs, dealt round: c, c + grid, ...
                for (int id = chunk + lane * ctas; id < rows * kKvHeads; id += 32 * ctas) {
                    const int index = (id - chunk) / ctas;
                    const uint32_t row_context = __ldcg(context_lengths + row_base + id / kKvHeads);
                    if (index < kMaxListTasks) {
                        Task task;
                        task.context =
                            static_cast<int>(min(row_context, static_cast<uint32_t>(capacity_units) * kUnitTokens));
                        task.row = row_base + id / kKvHeads;
                        task.kv_head = id % kKvHeads;
                        task.part = 0;
                        task.last = 1;
                        task.unit_begin = 0;
                        task.units = units_of_context(row_context, capacity_units);
                        tasks[index] = task;
                    }
                    ++count;
                }
                count = static_cast<int>(__reduce_add_sync(0xffffffffu, count));
            } else {
                const Position low = chunk_begin(plan, chunk, ctas);
                const Position high = chunk_begin(plan, chunk + 1, ctas);
                // the pieces inside the chunk, in (row, kv head) order: 32 pairs at a time
#pragma unroll 1
                for (int base = 0; base < rows * kKvHeads; base += 32) {
                    const int r = (base + lane) / kKvHeads;
                    const int kv = (base + lane) % kKvHeads;
                    bool inside = false;
                    Position start = high, occupied = 0;
                    if (r < rows) {
                        occupied = first_unit[r + 1] - first_unit[r];
                        start = pair_position(plan, r, kv, first_unit[r], occupied);
                        inside = piece_inside(start, occupied, low, high);
                    }
                    const uint32_t found = __ballot_sync(0xffffffffu, inside);
                    const int index = count + __popc(found & ((1u << lane) - 1u));
                    if (inside && index < kMaxListTasks) {
                        const uint32_t row_context = __ldcg(context_lengths + row_base + r);
                        const int row_units = units_of_context(row_context, capacity_units);
                        const PlanPiece piece = piece_of_pair(plan, start, occupied, chunk, low, high, ctas);
                        Task task;
                        task.context =
                            static_cast<int>(min(row_context, static_cast<uint32_t>(capacity_units) * kUnitTokens));
                        task.row = row_base + r;
                        task.kv_head = kv;
                        task.part = piece.part;
                        task.last = piece.last;
                        task.unit_begin = piece.begin;
                        task.units = max(0, min(piece.end, row_units) - piece.begin);
                        tasks[index] = task;
                    }
                    count += __popc(found);
                    if (__all_sync(0xffffffffu, start >= high)) {
                        break;
                    }
                }
            }
            __syncwarp();
            if (rehearsal) {
                break;
            }
            if (count > kMaxListTasks) {
                // cannot happen while the launcher's check of rows against the SM count holds
                if (lane == 0) {
                    atomicCAS(status, 0, kStatusAttentionPlanOverflow);
                }
                count = -1;
            }
            if (lane == 0) {
                sm.task_count[m & 1] = count;
                mbar_arrive(&sm.list_ready[m & 1]);
            }
            __syncwarp();
            if (count < 0) {
                break;
            }
            // The next chunk is claimed once the last bytes of this one have been asked for (an answer takes 0.2
            // us, the ring holds three stages); what lies past the end of the line is claimed too (it would
            // start, and find nothing to do).  Where no small chunk has work, because the tables describe far more
            // than the contexts take, there is nothing to wait for: the claims only clear the rest of the grid away,
            // and the sooner that is done, the sooner the merge kernel may start (nine rows in [128, 2048] under
            // tables of 32768 tokens 13.07 -> 12.92 us, as with a grid of one CTA per SM).
            chunk = -1;
            ok = att_wait(&sm.list_free[(m + 1) & 1], (((m + 1) >> 1) & 1) ^ 1, sm, status);
            if (ok && gridDim.x > ctas && chunk_begin(plan, ctas, ctas) < plan.line) {
                ok = att_wait(&sm.list_wanted, m & 1, sm, status);
            }
            while (gridDim.x > ctas && ok) {
                if (lane == 0) {
                    fence_proxy_async();  // the answer before this one has been read
                    mbar_arrive_expect_tx(&sm.claim_ready, 16);
                    claim_chunk(&sm.claim, &sm.claim_ready);
                }
                __syncwarp();
                ok = att_wait(&sm.claim_ready, claims & 1, sm, status);
                ++claims;
                chunk = ok ? claimed_chunk(&sm.claim) : -1;
                __syncwarp();
                if (chunk < 0 || chunk_begin(plan, chunk, ctas) < plan.line) {
                    break;
                }
            }
        }
    }

    if (warp == kKeyWarp || warp == kValueWarp) {
        // ---------------- K or V: two lanes per unit, one for each half of the dims -----------------
        const bool keys = warp == kKeyWarp;
        uint64_t* const full = keys ? sm.k_full : sm.v_full;
        uint64_t* const empty = keys ? sm.k_empty : sm.v_empty;
        uint8_t* const ring = keys ? &sm.k[0][0] : &sm.v[0][0];
        const CUtensorMap* const map = keys ? &key_map : &value_map;
        const int unit = lane >> 1;
        const int half = lane & 1;
        pdl_wait();
        for (int m = 0; ok; ++m) {
            ok = att_wait(&sm.list_ready[m & 1], (m >> 1) & 1, sm, status);
            const int count = ok ? sm.task_count[m & 1] : -1;
            if (count < 0) {
                break;
            }
            for (int i = 0; i < count && ok; ++i) {
                const Task task = sm.tasks[m & 1][i];
                const uint32_t* table = block_tables + static_cast<size_t>(task.row) * max_blocks;
                const int stages = (task.units + kStageUnits - 1) / kStageUnits;
                for (int st = 0; st < stages; ++st, ++n) {
                    const int slot = n % kStages;
                    const int first = task.unit_begin + st * kStageUnits;
                    const int units = min(kStageUnits, task.units - st * kStageUnits);
                    // the page id is fetched before the wait for a free slot, which is the longer of the two
                    const uint32_t physical = unit < units ? table[(first + unit) / units_per_page] : 0u;
                    ok = att_wait(&empty[slot], ((n / kStages) & 1) ^ 1, sm, status);
                    if (!ok) {
                        break;
                    }
                    // V that a partly filled stage leaves out is multiplied by probabilities of zero and must be
                    // finite, whatever the stage before it held: boxes in front of the first row arrive as zeros.  (The
                    // ring used to be cleared at the start of every CTA: 24 rows of at most 192 tokens 12.95 -> 12.68
                    // us, 32 rows in [128, 2048] 23.9 -> 23.6.)
                    const int boxes = keys ? units : kStageUnits;
                    if (lane == 0) {
                        mbar_arrive_expect_tx(&full[slot], static_cast<uint32_t>(boxes) * 2 * kBoxBytes);
                        if (keys) {
                            *reinterpret_cast<volatile int*>(&sm.stages_asked) = n + 1;
                        }
                    }
                    __syncwarp();
                    if (unit < boxes) {
                        const int row = unit < units ? (static_cast<int>(physical) * kKvHeads + task.kv_head) * page_size +
                                                           (first + unit) % units_per_page * kUnitTokens
                                                     : -kUnitTokens;
                        tma_box_g2s(ring + slot * kStageBytes + half * kHalfBytes + unit * kBoxBytes, map, half * 128, row,
                                    &full[slot]);
                    }
                    __syncwarp();
                }
            }
            __syncwarp();
            if (lane == 0 && ok) {
                if (keys) {
                    mbar_arrive(&sm.list_wanted);
                }
                mbar_arrive(&sm.list_free[m & 1]);
            }
        }
    } else if (warp == kMmaWarp) {
        // ---------------- tensor-core issue ---------------------------------------------------
        const uint32_t idesc_scores = (1u << 4) | (static_cast<uint32_t>(kColumns >> 3) << 17) | (8u << 24);
        const uint32_t idesc_output = idesc_scores | (1u << 15) | (1u << 16);  // both operands MN-major
        const uint32_t k_base = smem_u32(&sm.k[0][0]), v_base = smem_u32(&sm.v[0][0]);
        const uint32_t q_base = smem_u32(&sm.q[0][0]), p_base = smem_u32(&sm.p[0][0]);
        // O of stage m
        const auto issue_output = [&](int m) {
            const int slot = m % kStages;
            const int buffer = m & 1;
            const bool ready = att_wait(&sm.p_ready[buffer], (m >> 1) & 1, sm, status) &&
                               att_wait(&sm.v_full[slot], (m / kStages) & 1, sm, status) &&
                               att_wait(&sm.o_free[buffer], ((m >> 1) & 1) ^ 1, sm, status);
            if (!ready) {
                return false;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (elect_one()) {
#pragma unroll
                for (int half = 0; half < 2; ++half) {
                    const uint32_t d = tmem_base + kOutputColumn + (2 * buffer + half) * kColumns;
#pragma unroll
                    for (int ks = 0; ks < kStageTokens / 32; ++ks) {
                        // 32 tokens: four atoms of V; P: columns in chunks of 16, a chunk's tokens 16 bytes apart
                        umma_fp8(d, swizzled_descriptor(v_base + slot * kStageBytes + half * kHalfBytes + ks * 4096),
                                 smem_descriptor(p_base + buffer * kProbabilityBytes + ks * 512, 128, kStageTokens * 16),
                                 idesc_output, ks > 0 ? 1u : 0u);
                    }
                }
                umma_commit(&sm.v_empty[slot]);
                umma_commit(&sm.p_free[buffer]);
                umma_commit(&sm.o_ready[buffer]);
                mbar_arrive(&sm.o_ready[buffer]);
            }
            __syncwarp();
            return true;
        };
        for (int m = 0; ok; ++m) {
            ok = att_wait(&sm.list_ready[m & 1], (m >> 1) & 1, sm, status);
            const int count = ok ? sm.task_count[m & 1] : -1;
            if (count < 0) {
                break;
            }
            for (int i = 0; i < count && ok; ++i) {
                const int stages = (sm.tasks[m & 1][i].units + kStageUnits - 1) / kStageUnits;
                ok = att_wait(&sm.q_ready[t & 1], (t >> 1) & 1, sm, status);
                for (int st = 0; st < stages && ok; ++st) {
                    const int slot = n % kStages;
                    const int buffer = n & 1;
                    ok = att_wait(&sm.k_full[slot], (n / kStages) & 1, sm, status) &&
                         att_wait(&sm.s_free[buffer], ((n >> 1) & 1) ^ 1, sm, status);
                    if (!ok) {
                        break;
                    }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    if (elect_one()) {
                        const uint32_t d = tmem_base + kScoreColumn + buffer * kColumns;
#pragma unroll
                        for (int half = 0; half < 2; ++half) {
#pragma unroll
                            for (int ks = 0; ks < 4; ++ks) {
                                umma_fp8(d, swizzled_descriptor(k_base + slot * kStageBytes + half * kHalfBytes + ks * 32),
                                         smem_descriptor(q_base + (t & 1) * kQueryBytes + (half * 4 + ks) * 32 * kColumns,
                                                         kColumns * 16, 128),
                                         idesc_scores, (half > 0 || ks > 0) ? 1u : 0u);
                            }
                        }
                        umma_commit(&sm.k_empty[slot]);
                        if (st == stages - 1) {
                            umma_commit(&sm.q_free[t & 1]);
                        }
                        umma_commit(&sm.s_ready[buffer]);
                    }
                    __syncwarp();
                    ++n;
                    if (issued < n - 1) {
                        ok = issue_output(issued);
                        issued += ok ? 1 : 0;
                    }
                }
                if (stages == 0 && ok) {
                    // Nothing to multiply.  What is pending goes now: after a few tasks like this one the next query
                    // waits for the softmax warps, they for the output warps, and these for it.
                    if (issued < n) {
                        ok = issue_output(issued);
                        issued += ok ? 1 : 0;
                    }
                    if (lane == 0) {
                        mbar_arrive(&sm.q_free[t & 1]);
                    }
                    __syncwarp();
                }
                ++t;
            }
            // (the next chunk may be a while in coming)
            if (ok && issued < n) {
                ok = issue_output(issued);
                issued += ok ? 1 : 0;
            }
            __syncwarp();
            if (lane == 0 && ok) {
                mbar_arrive(&sm.list_free[m & 1]);
            }
        }
    } else if (warp < kSoftmaxWarps) {
        // ---------------- softmax: thread = token ---------------------------------------------
        const uint32_t s_lane = tmem_base + (static_cast<uint32_t>(warp * 32) << 16) + kScoreColumn;
        const int token = threadIdx.x;
        pdl_wait();
        for (int m = 0; ok; ++m) {
            ok = att_wait(&sm.list_ready[m & 1], (m >> 1) & 1, sm, status);
            const int count = ok ? sm.task_count[m & 1] : -1;
            if (count < 0) {
                break;
            }
            for (int i = 0; i < count && ok; ++i) {
                const Task task = sm.tasks[m & 1][i];
                const int stages = (task.units + kStageUnits - 1) / kStageUnits;
                ok = att_wait(&sm.q_ready[t & 1], (t >> 1) & 1, sm, status);
                if (!ok) {
                    break;
                }
                const float k_scale = key_scales ? key_scales[task.kv_head] : 1.0f;
                float score_scale[kGqaGroup], running_max[kGqaGroup], running_sum[kGqaGroup];
#pragma unroll
                for (int h = 0; h < kGqaGroup; ++h) {
                    score_scale[h] = softmax_scale * k_scale * kLog2e * sm.query_scale[t & 1][h];
                    running_max[h] = -INFINITY;  // log2 domain, the same in all threads
                    running_sum[h] = 0.0f;       // this thread's tokens only
                }
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive(&sm.q_free[t & 1]);  // (the scales have been read)
                }
                for (int st = 0; st < stages; ++st, ++n) {
                    const int buffer = n & 1;
                    const uint32_t parity = (n >> 1) & 1;
                    ok = att_wait(&sm.s_ready[buffer], parity, sm, status);
                    if (!ok) {
                        break;
                    }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    uint32_t d01[16], d23[16];
                    tmem_load16_issue(s_lane + buffer * kColumns, d01);
                    tmem_load16_issue(s_lane + buffer * kColumns + 16, d23);
                    tmem_load_wait();
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) {
                        mbar_arrive(&sm.s_free[buffer]);
                    }
                    const bool valid = (task.unit_begin + st * kStageUnits) * kUnitTokens + token < task.context &&
                                       token < (task.units - st * kStageUnits) * kUnitTokens;
                    float score[kGqaGroup];
                    float mine = -INFINITY;
#pragma unroll
                    for (int h = 0; h < kGqaGroup; ++h) {
                        score[h] = valid ? combine_query_digits(d01[h], d01[8 + h], d23[h], d23[8 + h]) * score_scale[h]
                                         : -INFINITY;
                        const float highest = warp_highest(score[h]);
                        mine = lane == h ? highest : mine;
                    }
                    if (lane < 8) {
                        sm.warp_max[buffer][warp][lane] = mine;
                    }
                    __syncwarp();
                    if (lane == 0) {
                        mbar_arrive(&sm.max_ready[buffer]);
                    }
                    ok = att_wait(&sm.max_ready[buffer], parity, sm, status);
                    if (!ok) {
                        break;
                    }
                    float probability[kGqaGroup], factor[kGqaGroup];
#pragma unroll
                    for (int h = 0; h < kGqaGroup; ++h) {
                        float new_max = running_max[h];
#pragma unroll
                        for (int w = 0; w < kSoftmaxWarps; ++w) {
                            new_max = fmaxf(new_max, sm.warp_max[buffer][w][h]);
                        }
                        factor[h] = new_max == -INFINITY ? 1.0f : exp2f(running_max[h] - new_max);
                        probability[h] = new_max == -INFINITY ? 0.0f : exp2f(score[h] - new_max);
                        running_sum[h] = fmaf(running_sum[h], factor[h], probability[h]);
                        running_max[h] = new_max;
                        probability[h] *= 256.0f;
                    }
                    uint32_t words[2 * kProbabilityDigits];
#pragma unroll
                    for (int j = 0; j < kProbabilityDigits; ++j) {
                        const uint32_t pair0 = take_digit(probability[0], probability[1]);
                        const uint32_t pair1 = take_digit(probability[2], probability[3]);
                        words[2 * j] = pair0 | pair1 << 16;
                        words[2 * j + 1] = take_digit(probability[4], probability[5]);
                    }
                    ok = att_wait(&sm.p_free[buffer], parity ^ 1, sm, status);
                    if (!ok) {
                        break;
                    }
                    *reinterpret_cast<uint4*>(&sm.p[buffer][token * 16]) = make_uint4(words[0], words[1], words[2], words[3]);
                    *reinterpret_cast<uint4*>(&sm.p[buffer][(kStageTokens + token) * 16]) = make_uint4(words[4], words[5], 0u, 0u);
                    // (four buffers: these words of stage n + 4 come after O of stage n + 2, which comes after the
                    // output warps have read stage n)
                    if (token == 0) {
#pragma unroll
                        for (int h = 0; h < kGqaGroup; ++h) {
                            sm.rescale[n & 3][h] = factor[h];
                        }
                    }
                    fence_proxy_async();
                    __syncwarp();
                    if (lane == 0) {
                        mbar_arrive(&sm.p_ready[buffer]);
                    }
                }
                if (!ok) {
                    break;
                }
                ok = att_wait(&sm.t_free[t & 1], ((t >> 1) & 1) ^ 1, sm, status);
                if (!ok) {
                    break;
                }
                float mine = 0.0f;
#pragma unroll
                for (int h = 0; h < kGqaGroup; ++h) {
                    const float sum = warp_sum(running_sum[h]);
                    mine = lane == h ? sum : mine;
                    if (token == 0) {
                        sm.task_max[t & 1][h] = running_max[h];
                    }
                }
                if (lane < 8) {
                    sm.task_sum[t & 1][warp][lane] = mine;
                }
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive(&sm.t_ready[t & 1]);
                }
                ++t;
            }
            __syncwarp();
            if (lane == 0 && ok) {
                mbar_arrive(&sm.list_free[m & 1]);
            }
        }
    } else if (warp >= kFirstQueryWarp && warp < kPlanWarp) {
        // ---------------- query digits: half of the heads per warp, eight dims per lane --------------
        // (A task cannot start before they are there, so two warps share them, and no branch keeps one head's
        // conversions from running beside another's.  Us per layer, one warp with three digits in fp32 / with four /
        // two warps with four in f16: one row of 2048 12.2 / 12.7 / 11.2, 32 rows in [128, 2048] 25.1 / 27.4 / 24.3; the
        // last two digits only for heads that need them: 11.1 and 24.3.)
        constexpr int kHeads = kGqaGroup / kQueryWarps;
        const int first_head = (warp - kFirstQueryWarp) * kHeads;
        pdl_wait();
        for (int m = 0; ok; ++m) {
            ok = att_wait(&sm.list_ready[m & 1], (m >> 1) & 1, sm, status);
            const int count = ok ? sm.task_count[m & 1] : -1;
            if (count < 0) {
                break;
            }
            for (int i = 0; i < count && ok; ++i) {
                const Task task = sm.tasks[m & 1][i];
                const uint2* at_lane = reinterpret_cast<const uint2*>(
                    query +
                    (static_cast<size_t>(task.row) * kQueryHeads + task.kv_head * kGqaGroup + first_head) * kHeadDim +
                    8 * lane);
                uint32_t pairs[kHeads][4];  // (rows start on 8-byte boundaries)
#pragma unroll
                for (int h = 0; h < kHeads; ++h) {
                    const uint2 first = at_lane[h * (kHeadDim / 4)];
                    const uint2 second = at_lane[h * (kHeadDim / 4) + 1];
                    pairs[h][0] = first.x;
                    pairs[h][1] = first.y;
                    pairs[h][2] = second.x;
                    pairs[h][3] = second.y;
                }
                ok = att_wait(&sm.q_free[t & 1], ((t >> 1) & 1) ^ 1, sm, status);
                if (!ok) {
                    break;
                }
                uint32_t digits[kHeads][kQueryDigits][4];
#pragma unroll
                for (int h = 0; h < kHeads; ++h) {
                    uint32_t highest = 0;
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        highest = max(highest, max(pairs[h][j] & 0x7fffu, (pairs[h][j] >> 16) & 0x7fffu));
                    }
                    highest = __reduce_max_sync(0xffffffffu, highest);
                    // largest magnitude to [128, 256).  With an infinity in the head only the infinities count, and
                    // the scores become infinities (or NaN) when they are scaled back; a NaN is an e4m3 NaN.
                    const uint32_t exponent = max(highest >> 7, 8u);
                    const bool infinite = highest >= 0x7f80u;
                    const float up = __uint_as_float((261u - exponent) << 23);
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        float lo = __uint_as_float(pairs[h][j] << 16), hi = __uint_as_float(pairs[h][j] & 0xffff0000u);
                        if (infinite) {
                            lo = isnan(lo) ? lo : isinf(lo) ? copysignf(1.0f, lo) : 0.0f;
                            hi = isnan(hi) ? hi : isinf(hi) ? copysignf(1.0f, hi) : 0.0f;
                        } else {
                            lo *= up;
                            hi *= up;
                        }
                        take_high_digits(lo, hi, digits[h][0][j], digits[h][1][j]);
                        take_low_digits(lo, hi, digits[h][0][j], digits[h][1][j], digits[h][2][j], digits[h][3][j]);
                    }
                    if (lane == 0) {
                        sm.query_scale[t & 1][first_head + h] =
                            infinite ? INFINITY : __uint_as_float((exponent - 7u) << 23);
                    }
                }
                uint8_t* const at = &sm.q[t & 1][(lane >> 1) * 16 * kColumns + first_head * 16 + (lane & 1) * 8];
#pragma unroll
                for (int h = 0; h < kHeads; ++h) {
#pragma unroll
                    for (int d = 0; d < kQueryDigits; ++d) {
                        *reinterpret_cast<uint2*>(at + h * 16 + d * 128) = make_uint2(
                            digits[h][d][0] | digits[h][d][1] << 16, digits[h][d][2] | digits[h][d][3] << 16);
                    }
                }
                fence_proxy_async();
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive(&sm.q_ready[t & 1]);
                }
                ++t;
            }
            __syncwarp();
            if (lane == 0 && ok) {
                mbar_arrive(&sm.list_free[m & 1]);
            }
        }
    } else if (warp < kMmaWarp) {
        // ---------------- outputs: thread = dim -----------------------------------------------
        const int o_warp = warp - kFirstOutputWarp;
        const int half = o_warp >> 2;
        const int dim = half * 128 + (o_warp & 3) * 32 + lane;
        const uint32_t o_lane = tmem_base + (static_cast<uint32_t>((o_warp & 3) * 32) << 16) + kOutputColumn + half * kColumns;
        pdl_wait();
        for (int m = 0; ok; ++m) {
            ok = att_wait(&sm.list_ready[m & 1], (m >> 1) & 1, sm, status);
            const int count = ok ? sm.task_count[m & 1] : -1;
            if (count < 0) {
                break;
            }
            for (int i = 0; i < count && ok; ++i) {
                const Task task = sm.tasks[m & 1][i];
                const int row = task.row;
                const int kv_head = task.kv_head;
                const int stages = (task.units + kStageUnits - 1) / kStageUnits;
                float total[kGqaGroup];
#pragma unroll
                for (int h = 0; h < kGqaGroup; ++h) {
                    total[h] = 0.0f;
                }
                for (int st = 0; st < stages; ++st, ++n) {
                    const int buffer = n & 1;
                    ok = att_wait(&sm.o_ready[buffer], (n >> 1) & 1, sm, status);
                    if (!ok) {
                        break;
                    }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    uint32_t d01[16], d2[8];
                    tmem_load16_issue(o_lane + 2 * buffer * kColumns, d01);
                    tmem_load8_issue(o_lane + 2 * buffer * kColumns + 16, d2);
                    float factor[kGqaGroup];
#pragma unroll
                    for (int h = 0; h < kGqaGroup; ++h) {
                        factor[h] = sm.rescale[n & 3][h];
                    }
                    tmem_load_wait();
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) {
                        mbar_arrive(&sm.o_free[buffer]);
                    }
#pragma unroll
                    for (int h = 0; h < kGqaGroup; ++h) {
                        total[h] = fmaf(total[h], factor[h], combine_digits(d01[h], d01[8 + h], d2[h]));
                    }
                }
                if (!ok) {
                    break;
                }
                ok = att_wait(&sm.t_ready[t & 1], (t >> 1) & 1, sm, status);
                if (!ok) {
                    break;
                }
                // (the probabilities were multiplied with 256)
                const float v_scale = (value_scales ? value_scales[kv_head] : 1.0f) * 0.00390625f;
#pragma unroll
                for (int h = 0; h < kGqaGroup; ++h) {
                    float denominator = 0.0f;
#pragma unroll
                    for (int w = 0; w < kSoftmaxWarps; ++w) {
                        denominator += sm.task_sum[t & 1][w][h];
                    }
                    const float inverse = denominator > 0.0f ? v_scale / denominator : 0.0f;
                    const float value = total[h] * inverse;
                    const int head = kv_head * kGqaGroup + h;
                    const size_t pair = static_cast<size_t>(row - row_base) * kQueryHeads + head;
                    if (kSplit) {
                        const size_t slot = pair * partitions + task.part;
                        if (dim == 0) {
                            float* stats = partial_stats + slot * kPartialFloats;
                            stats[0] = sm.task_max[t & 1][h];
                            // the last piece of a pair carries a sign
                            stats[1] = task.last ? __uint_as_float(__float_as_uint(denominator) | 0x80000000u)
                                                 : fabsf(denominator);
                        }
                        partial_out[slot * kHeadDim + dim] = __float2half_rn(value);
                    } else {
                        float gated = value;
                        if (query_gate_projection != nullptr) {
                            const float gate = __bfloat162float(query_gate_projection[static_cast<size_t>(row) * gate_stride +
                                                                                      head * (2 * kHeadDim) + kHeadDim + dim]);
                            gated *= 1.0f / (1.0f + __expf(-gate));
                        }
                        const __nv_bfloat16 rounded = __float2bfloat16(gated);
                        if (output != nullptr) {
                            output[(static_cast<size_t>(row) * kQueryHeads + head) * kHeadDim + dim] = rounded;
                        }
                        if (staged_output != nullptr) {
                            // the same value as f16 in the operand layout of the output projection
                            const int feature = head * kHeadDim + dim;
                            staged_output[(static_cast<size_t>(feature >> 3) * padded_rows + row) * 8 + (feature & 7)] = bf16_to_f16(rounded);
                        }
                    }
                }
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive(&sm.t_free[t & 1]);
                }
                ++t;
            }
            __syncwarp();
            if (lane == 0 && ok) {
                mbar_arrive(&sm.list_free[m & 1]);
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (*reinterpret_cast<volatile int*>(&sm.failed) != 0) {
        // A wait gave up somewhere.  Whoever asked for something that arrives by itself waits for it, 0.2 ms at most for
        // each, whether its own waits went well or not: the memory it arrives in must still be this CTA's.
        const auto arrived = [](uint64_t* bar, int index, int ring) {
            const long long start = clock64();
            while (!mbar_try_wait(&bar[index % ring], (index / ring) & 1) && clock64() - start < 400000ll) {
            }
        };
        if (warp == kKeyWarp || warp == kValueWarp) {  // copies: the last trip round the ring
            for (int i = n > kStages ? n - kStages : 0; i < n; ++i) {
                arrived(warp == kKeyWarp ? sm.k_full : sm.v_full, i, kStages);
            }
        } else if (warp == kMmaWarp) {  // MMAs, to the last of their commits
            if (n > 0) {
                arrived(sm.s_ready, n - 1, 2);
            }
            if (issued > 0) {
                arrived(sm.o_ready, issued - 1, 2);
            }
        } else if (warp == kPlanWarp && claims > 0) {  // the answer to a claim
            arrived(&sm.claim_ready, claims - 1, 1);
        }
        __syncthreads();
    }
    if (warp == kMmaWarp) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kTmemColumns) : "memory");
    }
}

// Log-sum-exp merge of the partitions, output gate, bf16 store (as cuda/paged_attention.cu:1736-1823).
// One CTA per (row, head): the longest row of a ragged batch has dozens of partials, and a single warp walking them
// is a chain of dependent memory round trips.  Warp w takes the partials w, w + 8, ... (eight dims per lane), the
// sums meet in shared memory in warp order.  A pair's partials lie side by side and the sign of the sum marks the
// last one; the slots behind it were never written.  Statistics and outputs are asked for together, before that
// mark is known.  (The kernel used to make the
// attention kernel's plan again, a microsecond and a half of dependent arithmetic: from the end of the wait to the
// last store 4.4 us, now 1.6.)
constexpr int kMergeWarps = 8;
constexpr int kMergeDepth = 4;

__global__ void __launch_bounds__(kMergeWarps * 32) reduce_partitions_kernel(
    const float* __restrict__ partial_stats, const __half* __restrict__ partial_out,
    const __nv_bfloat16* __restrict__ query_gate_projection, __nv_bfloat16* __restrict__ output,
    __half* __restrict__ staged_output, int padded_rows, int partitions, int row_base, int gate_stride) {
    pdl_launch_dependents();  // the output projection may start streaming its weights
    __shared__ float sums[kMergeWarps][kHeadDim];
    __shared__ float denominators[kMergeWarps];
    const int pair = blockIdx.x;  // (row, head)
    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const int row = row_base + pair / kQueryHeads;
    const int head = pair % kQueryHeads;
    const float2* stats = reinterpret_cast<const float2*>(partial_stats) + static_cast<size_t>(pair) * partitions;
    const __half* outs = partial_out + static_cast<size_t>(pair) * partitions * kHeadDim + 8 * lane;
    pdl_wait();
    uint4 raw[kMergeDepth];
    float2 raw_stats[kMergeDepth];
    const auto fetch = [&](int first, int end) {
#pragma unroll
        for (int j = 0; j < kMergeDepth; ++j) {
            const int p = first + j * kMergeWarps;
            raw_stats[j] = make_float2(-INFINITY, 0.0f);
            raw[j] = make_uint4(0, 0, 0, 0);
            if (p < end) {
                raw_stats[j] = stats[p];
                raw[j] = *reinterpret_cast<const uint4*>(outs + static_cast<size_t>(p) * kHeadDim);
            }
        }
    };
    fetch(warp, partitions);
    // every warp looks for the last partial and finds the maximum over all of them (lanes side by side) ...
    float maximum = -INFINITY;
    int used = partitions;
    for (int base = 0; base < used; base += 32) {
        const float2 mine = base + lane < partitions ? stats[base + lane] : make_float2(-INFINITY, 0.0f);
        const uint32_t marks = __ballot_sync(0xffffffffu, (__float_as_uint(mine.y) >> 31) != 0);
        if (marks != 0) {
            used = base + __ffs(marks);
        }
        if (base + lane < used && fabsf(mine.y) > 0.0f) {
            maximum = fmaxf(maximum, mine.x);
        }
    }
    maximum = warp_highest(maximum);
    // ... and adds up its own
    float denominator = 0.0f;
    float acc[8] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
    for (int first = warp; first < used; first += kMergeDepth * kMergeWarps) {
        if (first != warp) {
            fetch(first, used);
        }
#pragma unroll
        for (int j = 0; j < kMergeDepth; ++j) {
            const float sum = fabsf(raw_stats[j].y);
            const bool present = first + j * kMergeWarps < used;
            const float weight = present && sum > 0.0f ? sum * exp2f(raw_stats[j].x - maximum) : 0.0f;
            denominator += weight;
            const __half2* h = reinterpret_cast<const __half2*>(&raw[j]);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float2 f = __half22float2(h[i]);
                if (present) {  // (a slot that was never written may hold anything)
                    acc[2 * i] += weight * f.x;
                    acc[2 * i + 1] += weight * f.y;
                }
            }
        }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        sums[warp][8 * lane + i] = acc[i];
    }
    if (lane == 0) {
        denominators[warp] = denominator;
    }
    __syncthreads();
    // a thread per dim
    const int dim = threadIdx.x;
    float total = 0.0f;
    denominator = 0.0f;
#pragma unroll
    for (int w = 0; w < kMergeWarps; ++w) {
        denominator += denominators[w];
        total += sums[w][dim];
    }
    const float inverse = denominator > 0.0f ? 1.0f / denominator : 0.0f;
    float gate = 1.0f;
    if (query_gate_projection != nullptr) {
        gate = __bfloat162float(
            query_gate_projection[static_cast<size_t>(row) * gate_stride + head * (2 * kHeadDim) + kHeadDim + dim]);
        gate = 1.0f / (1.0f + __expf(-gate));
    }
    const __nv_bfloat16 rounded = __float2bfloat16(total * inverse * gate);
    if (output != nullptr) {
        output[(static_cast<size_t>(row) * kQueryHeads + head) * kHeadDim + dim] = rounded;
    }
    if (staged_output != nullptr) {
        // the same value as f16 in the operand layout of the output projection
        const int feature = head * kHeadDim + dim;
        staged_output[(static_cast<size_t>(feature >> 3) * padded_rows + row) * 8 + (feature & 7)] = bf16_to_f16(rounded);
    }
}
static_assert(kMergeWarps * 32 == kHeadDim, "a thread per dim");

using AttentionKernel = void (*)(const CUtensorMap, const CUtensorMap, const __nv_bfloat16*, const __nv_bfloat16*,
                                 const uint32_t*, const uint32_t*, const float*, const float*, __nv_bfloat16*, __half*,
                                 int, float*, __half*, int, int, int, int, int, int, int, int, float, int*);
const AttentionKernel attention_kernels[3] = {paged_attention_packed_kernel<false, uint32_t>,
                                              paged_attention_packed_kernel<true, uint32_t>,
                                              paged_attention_packed_kernel<true, unsigned long long>};

cudaError_t launch_attention(const void* query, const void* query_gate_projection, const void* key_cache,
                             const void* value_cache, const void* block_tables, const void* context_lengths,
                             const float* key_scales, const float* value_scales, void* output, void* workspace,
                             size_t workspace_bytes, int rows, int row_base, int max_blocks, int page_size,
                             int gate_stride, int partitions, float softmax_scale, cudaStream_t stream,
                             void* staged_output = nullptr) {
    if (gate_stride == 0) {
        gate_stride = kQueryHeads * 2 * kHeadDim;
    }
    if (gate_stride < kQueryHeads * 2 * kHeadDim || gate_stride % 8 != 0) {
        return cudaErrorInvalidValue;
    }
    if (query == nullptr || key_cache == nullptr || value_cache == nullptr || block_tables == nullptr ||
        context_lengths == nullptr || (output == nullptr && staged_output == nullptr) ||
        (staged_output != nullptr && row_base + rows > 32) || rows <= 0 || rows > kPlanRows || row_base < 0 ||
        max_blocks <= 0 || partitions <= 0 || partitions > 65535 || !isfinite(softmax_scale) ||
        softmax_scale <= 0.0f || (page_size != 16 && page_size != 64)) {
        return cudaErrorInvalidValue;
    }
    int* status = status_ptr();
    if (status == nullptr) {
        return cudaErrorInvalidValue;
    }
    const size_t shared = sizeof(Smem) + 1024;
    static PerDevice<cudaError_t> opted_per_device;
    const cudaError_t* opted = opted_per_device.get([shared]() {
        for (const AttentionKernel kernel : attention_kernels) {
            const cudaError_t error =
                cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(shared));
            if (error != cudaSuccess) {
                return error;
            }
        }
        return cudaSuccess;
    });
    if (opted == nullptr) {
        return cudaErrorInvalidDevice;
    }
    if (*opted != cudaSuccess) {
        return *opted;
    }
    // One CTA per SM at a time, whatever the batch: the task lists are cut on the device.
    int device = 0, sms = 0;
    if (cudaGetDevice(&device) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess || sms <= 0) {
        return cudaErrorInvalidDevice;
    }
    if (!plan_fits(rows, sms)) {
        return cudaErrorInvalidValue;
    }
    CUtensorMap key_map, value_map;
    cudaError_t encoded = encode_cache_map(&key_map, key_cache);
    if (encoded == cudaSuccess) {
        encoded = encode_cache_map(&value_map, value_cache);
    }
    if (encoded != cudaSuccess) {
        return encoded;
    }
    const int padded_rows = row_base + rows <= 16 ? 16 : 32;  // of the staged output
    const bool split = partitions > 1;
    const size_t partials = static_cast<size_t>(rows) * kQueryHeads * partitions;
    if (split && (workspace == nullptr || workspace_bytes < partials * kPartialBytes)) {
        return cudaErrorInvalidValue;
    }
    // partials is a multiple of 24, so the f16 block starts on a 16-byte boundary.
    float* partial_stats = split ? static_cast<float*>(workspace) : nullptr;
    __half* partial_out = split ? reinterpret_cast<__half*>(partial_stats + partials * kPartialFloats) : nullptr;
    const PlanShape plan =
        split ? plan_shape(rows, max_blocks, page_size, partitions, sms) : PlanShape{0, false, false};
    const AttentionKernel kernel = attention_kernels[split ? (plan.wide ? 2 : 1) : 0];
    // (undivided rows: no CTA without a task; 24 rows of 128 tokens 6.23 -> 6.01 us)
    const int grid = !split ? std::min(sms, rows * kKvHeads) : plan.may_be_dynamic ? kChunksPerSm * sms : sms;
    const cudaError_t launched = qwc::launch_chained(
        kernel, dim3(grid), dim3(kThreads), shared, stream, key_map, value_map,
        static_cast<const __nv_bfloat16*>(query), static_cast<const __nv_bfloat16*>(query_gate_projection),
        static_cast<const uint32_t*>(block_tables), static_cast<const uint32_t*>(context_lengths), key_scales,
        value_scales, split ? nullptr : static_cast<__nv_bfloat16*>(output),
        split ? nullptr : static_cast<__half*>(staged_output), padded_rows, partial_stats, partial_out, rows, max_blocks,
        row_base, page_size, gate_stride, partitions, plan.smallest_chunk, sms, softmax_scale, status);
    if (launched != cudaSuccess || !split) {
        return launched;
    }
    return qwc::launch_chained(reduce_partitions_kernel, dim3(rows * kQueryHeads), dim3(kMergeWarps * 32), 0, stream,
                               partial_stats, partial_out, static_cast<const __nv_bfloat16*>(query_gate_projection),
                               static_cast<__nv_bfloat16*>(output), static_cast<__half*>(staged_output), padded_rows,
                               partitions, row_base, gate_stride);
}

// ---- built-in scratch for callers that cannot allocate ------------------------------------
//
// Split-context partials normally live in a workspace the caller allocates.  Some callers have
// no way to do that: a process that handed its whole VRAM budget out at start-up and refuses
// any later cudaMalloc (the reference engine enforces such a ceiling), a thin foreign-language
// binding that can pass pointers it was given but owns no device allocator, or a diagnostic
// attached to a running server.  For them the library carries its own scratch: a fixed array
// in device memory, sized for kStaticPartialPairs (row, partition) pairs.  It exists once per
// GPU that loads the library and stays resident until the process exits.
constexpr int kStaticPartialPairs = 512;  // rows * partitions, e.g. 32 rows x 16 partitions
constexpr size_t kStaticScratchBytes = static_cast<size_t>(kStaticPartialPairs) * kQueryHeads * kPartialBytes;
static __device__ __align__(256) unsigned char g_static_partials[kStaticScratchBytes];

// Device address of the array above for the current device.  In host code the symbol's name is
// only a handle, never an address a kernel may be given, so the address is asked of the runtime
// once per device (with that device current) and remembered.
cudaError_t static_partials_address(void** out) {
    constexpr int kMaxDevices = 64;
    static void* cached[kMaxDevices] = {};
    int device = 0;
    cudaError_t err = cudaGetDevice(&device);
    if (err != cudaSuccess) {
        return err;
    }
    if (device < 0 || device >= kMaxDevices) {
        return cudaErrorInvalidDevice;
    }
    if (cached[device] == nullptr) {
        void* address = nullptr;
        err = cudaGetSymbolAddress(&address, g_static_partials);
        if (err != cudaSuccess) {
            return err;
        }
        cached[device] = address;
    }
    *out = cached[device];
    return cudaSuccess;
}

}  // namespace
}  // namespace qwc

extern "C" size_t qwc_paged_attention_packed_workspace_bytes(int rows, int partitions) {
    if (rows <= 0 || partitions <= 1) {
        return 0;
    }
    return static_cast<size_t>(rows) * qwc::kQueryHeads * partitions * qwc::kPartialBytes;
}

extern "C" int qwc_paged_attention_packed_fp8(const void* query, const void* query_gate_projection,
                                              const void* key_cache, const void* value_cache,
                                              const void* block_tables, const void* context_lengths, void* output,
                                              void* workspace, size_t workspace_bytes, int rows, int row_base,
                                              int max_blocks, int tile_size, int partitions, float softmax_scale,
                                              cudaStream_t stream) {
    if (tile_size <= 0 || tile_size > 64) {
        return cudaErrorInvalidValue;
    }
    if (tile_size != qwc::kGqaGroup) {
        return cudaErrorNotSupported;  // segment tiles are prefill shapes
    }
    return qwc::launch_attention(query, query_gate_projection, key_cache, value_cache, block_tables,
                                 context_lengths, nullptr, nullptr, output, workspace, workspace_bytes, rows,
                                 row_base, max_blocks, qwc::current_shape().kv_page_size, 0, partitions,
                                 softmax_scale, stream);
}

extern "C" int qwc_paged_attention_packed_fp8_scaled(const void* query, const void* query_gate_projection,
                                                     const void* key_cache, const void* value_cache,
                                                     const void* block_tables, const void* context_lengths,
                                                     const float* key_scales, const float* value_scales,
                                                     void* output, void* workspace, size_t workspace_bytes,
                                                     int rows, int row_base, int max_blocks, int page_size,
                                                     int gate_stride, int partitions, float softmax_scale,
                                                     cudaStream_t stream) {
    return qwc::launch_attention(query, query_gate_projection, key_cache, value_cache, block_tables,
                                 context_lengths, key_scales, value_scales, output, workspace, workspace_bytes,
                                 rows, row_base, max_blocks, page_size, gate_stride, partitions, softmax_scale,
                                 stream);
}

extern "C" int qwc_paged_attention_packed_fp8_staged(const void* query, const void* query_gate_projection,
                                                     const void* key_cache, const void* value_cache,
                                                     const void* block_tables, const void* context_lengths,
                                                     const float* key_scales, const float* value_scales,
                                                     void* output, void* staged_output, void* workspace,
                                                     size_t workspace_bytes, int rows, int row_base, int max_blocks,
                                                     int page_size, int gate_stride, int partitions,
                                                     float softmax_scale, cudaStream_t stream) {
    return qwc::launch_attention(query, query_gate_projection, key_cache, value_cache, block_tables,
                                 context_lengths, key_scales, value_scales, output, workspace, workspace_bytes,
                                 rows, row_base, max_blocks, page_size, gate_stride, partitions, softmax_scale,
                                 stream, staged_output);
}

extern "C" int qwc_paged_attention_packed_fp8_noalloc(const void* query, const void* query_gate_projection,
                                                      const void* key_cache, const void* value_cache,
                                                      const void* block_tables, const void* context_lengths,
                                                      const float* key_scales, const float* value_scales,
                                                      void* output, int rows, int row_base, int max_blocks,
                                                      int page_size, int gate_stride, int partitions,
                                                      float softmax_scale, cudaStream_t stream) {
    if (rows <= 0 || partitions <= 0) {
        return cudaErrorInvalidValue;
    }
    // The built-in scratch holds kStaticPartialPairs (row, partition) pairs and not one more.
    if (static_cast<long long>(rows) * partitions > qwc::kStaticPartialPairs) {
        return cudaErrorInvalidValue;
    }
    void* scratch = nullptr;
    const cudaError_t resolved = qwc::static_partials_address(&scratch);
    if (resolved != cudaSuccess) {
        return resolved;
    }
    // Nothing needs clearing first.  The merge loads statistics and outputs of slots that this call may not have
    // written, but what it uses ends at the last piece of a pair, which the sign of its sum marks: the pieces of a
    // pair lie side by side from slot 0 on, and all of them are written by every call.
    return qwc::launch_attention(query, query_gate_projection, key_cache, value_cache, block_tables,
                                 context_lengths, key_scales, value_scales, output, scratch,
                                 qwc::kStaticScratchBytes, rows, row_base, max_blocks, page_size, gate_stride,
                                 partitions, softmax_scale, stream);
}

extern "C" int qwc_paged_attention_packed_noalloc_max_pairs(void) { return qwc::kStaticPartialPairs; }
