// NVFP4 projections of up to eight activation rows with both operands in four bits: the weights go
// from memory to the tensor cores as they are stored (tcgen05.mma.kind::mxf4nvf4, e2m1 values and e4m3
// scales of 16), and an activation enters as eight e2m1 digits, one column of the B operand each.
//
// What the f16 kernels (nvfp4_umma.cu, nvfp4_streamk.cu) spend their time on at these batches is widening
// weights: one conversion per two weights keeps the conversion unit 70 % busy, a stage takes as long as
// its bytes need from HBM, and the stages in the ring are still to be widened when the last byte has
// landed.  Here nobody touches a weight: the end of the launch follows the last byte, and what bounds the
// kernel is the weight stream, between a start and a tail of about 3 us.  Measured (us, bf16 rows in, layers
// that L2 does not hold, a dozen different activations, f16 / four bits at one and at eight rows): 34816 x 5120
// 22.8 / 18.9 (5.3 TB/s) and 21.0 / 20.4, 5120 x 17408 15.7 / 12.8 and 16.3 / 15.4, 5120 x 6144 10.9 / 7.8 and
// 11.1 / 9.7.
//
// Not above eight rows, and not for staged activations inside a decode step: making digits costs about 25
// instructions per activation in every CTA, after the activations have arrived.  At sixteen rows that
// takes longer than the weights (34816 x 5120: 30.3 us against 24.6), and in a step it lies between the
// norm and the first MMA of every projection (one row: the step 4.58 -> 4.82 ms, although the projections
// alone went from 3.09 to 2.99 ms).
//
// Digits.  The sixteen activations of a block (16 features of one row) share a power of two; each is
// written as 23 bits of fixed point below it, in balanced base 8 (digits -4 .. 4, which are e2m1 values),
// and digit j of row r becomes column j R + r of the B operand (R: rows padded to a power of two).  The sum
// over K of every column is an fp32 accumulator of its own, and the epilogue adds the eight with their
// weights 8^(j - 7).  An activation arrives as the f16 that the other kernels multiply with, here with the
// eight significant bits of a bf16: the 23 bits hold it exactly unless it is 2^-14 times smaller than its
// block's power of two.  A warp that meets such a one (N(0, 1) activations: one warp and stage in thirty)
// writes what is left of its activations as eight digits more, 2^-23 times smaller, and they are multiplied
// into accumulators of their own; a launch with such a warp somewhere takes 0.1 to 0.9 us longer, and nobody
// else pays.  Together they reach from f16's largest to its smallest bit: both operands
// are exact, as they are in the f16 kernels, and only the sums are rounded.  That can be seen where the exact
// result is 0 (every block of features twice, with opposite weights, shuffled over K = 4096): outputs of
// 3.4e-8 of the uncancelled sums, 1.3e-7 on the f16 kernel.
//
//   warp 0      weight producer: two boxes of 128 rows x 128 bytes and their scale blocks per stage
//   warp 1      copies the stage's scales to tensor memory (tcgen05.cp) and issues the MMAs
//   warps 2-3   look at the stage's scale bytes: the tensor cores take them as unsigned, so a block whose
//               scale is negative has the sign moved into its sixteen values
//   warps 4-11  turn activations into digits (a lane per block), then read the accumulators, combine, store
//
// Every wait is bounded, as in nvfp4_streamk.cu.
#pragma once

namespace qwc {
namespace {

constexpr int kNativeRows = 8;                   // activation rows at most
constexpr int kNativeDigits = 8;
constexpr int kNativeWorkerWarps = 8;
constexpr int kNativeFirstWorker = 4;
constexpr int kNativeThreads = (kNativeFirstWorker + kNativeWorkerWarps) * 32;
constexpr int kNativeXBytes = 4 * (2 * kNativeRows * kNativeDigits * 128 + 2048);  // ring of digit tiles
constexpr int kNativeMaxXSlots = 8;
constexpr int kNativeSmemBytes = kWeightStages * kTiles * kTileStageBytes + kNativeXBytes + 1024;
constexpr int kNativeAccumulator = 128;          // columns of one tile's accumulators ...
constexpr int kNativeRest = 64;                  // ... of which those of the second eight digits start here
constexpr int kNativeScaleColumn = 256;          // tensor memory behind the accumulators: scales
constexpr int kNativeScaleColumns = 48;          // of one stage: 16 per tile, 16 for the activations

struct NativeBarriers {
    uint64_t w_full[kWeightStages];
    uint64_t w_checked[kWeightStages];
    uint64_t w_empty[kWeightStages];
    uint64_t x_full[kNativeMaxXSlots];
    uint64_t x_empty[kNativeMaxXSlots];
    uint64_t done;
    uint32_t tmem_base;
    uint32_t rest[kNativeMaxXSlots];  // byte w: warp w of the slot's team wrote the second eight digits
    int rest_used;
    int failed;
};

__device__ __noinline__ bool native_wait_slow(uint64_t* bar, uint32_t parity, NativeBarriers* b, int* status) {
    const long long start = clock64();
    for (;;) {
#pragma unroll 1
        for (int spin = 0; spin < 64; ++spin) {
            if (mbar_try_wait(bar, parity)) {
                return true;
            }
        }
        if (*reinterpret_cast<volatile int*>(&b->failed) != 0) {
            return false;
        }
        if (clock64() - start > 40000000ll) {
            break;
        }
    }
    atomicCAS(status, 0, kStatusGemvWait);
    *reinterpret_cast<volatile int*>(&b->failed) = 1;
    return false;
}

// For a converged warp: the same answer in every lane.
__device__ __forceinline__ bool native_wait(uint64_t* bar, uint32_t parity, NativeBarriers* b, int* status) {
    const bool ok = mbar_try_wait(bar, parity) || native_wait_slow(bar, parity, b, status);
    return __all_sync(0xffffffffu, ok);
}

// K-major operand whose rows are 128 bytes with the 128-byte swizzle, eight rows (1 KiB) to an atom.
__device__ __forceinline__ uint64_t swizzled_descriptor(uint32_t address) {
    const uint64_t lo = ((address >> 4) & 0x3FFFu) | (1ull << 16);
    const uint64_t hi = (1024u >> 4) | (1u << 14) | (2u << 29);
    return lo | (hi << 32);
}

// D[128][N] (+)= A[128][64] x B[N][64], e2m1 with an e4m3 scale per 16; scales in tensor memory.
__device__ __forceinline__ void umma_nvfp4(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                           uint32_t scale_a, uint32_t scale_b, uint32_t accumulate) {
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "setp.ne.b32 p, %6, 0;\n"
        "tcgen05.mma.cta_group::1.kind::mxf4nvf4.block_scale.scale_vec::4X [%0], %1, %2, %3, [%4], [%5], p;\n"
        "}\n" ::"r"(d_tmem),
        "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(scale_a), "r"(scale_b), "r"(accumulate)
        : "memory");
}

// 512 bytes (32 rows of 16) to four columns of tensor memory, the same in all four lane quarters.
__device__ __forceinline__ void copy_scales(uint32_t tmem, uint64_t desc) {
    asm volatile("tcgen05.cp.cta_group::1.32x128b.warpx4 [%0], %1;" ::"r"(tmem), "l"(desc) : "memory");
}

// (.aligned: the whole warp at once, and every warp gets here from a region that ends with one lane at work)
__device__ __forceinline__ void native_cluster_sync() {
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// A word of another CTA of the cluster, at the place where this CTA has `local`.
__device__ __forceinline__ uint32_t native_peer_word(const void* local, int rank) {
    uint32_t remote, value;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(smem_u32(local)), "r"(rank));
    asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(value) : "r"(remote) : "memory");
    return value;
}

__device__ __forceinline__ float native_peer_float(const float* local, int rank) {
    return __uint_as_float(native_peer_word(local, rank));
}

// The 2^23 binade, whose low bits are the integer that was added, and what turns them into the integer plus 4 in
// every octal digit.
constexpr float kBinade = 12582912.0f;
constexpr uint32_t kToOctal = 0x924924u - 0x4B400000u;

// Eight digits + 4 -> e2m1: below 4 the sign bit and 4 - digit, from 4 on digit - 4 (codes 0 .. 4 are 0, 0.5,
// .. 2).  `first`: the first digits of numbers, which go up to 4.
__device__ __forceinline__ uint32_t e2m1_digits(uint32_t octal, bool first) {
    const uint32_t four = first ? (octal & 0x88888888u) >> 1 : 0u;
    const uint32_t negative = (~(octal | four) & 0x44444444u) >> 2;
    return (((octal ^ (3u * negative)) & 0x33333333u) | four) + 9u * negative;
}

// Eight e2m1 digits of sixteen numbers (each an integer plus 4 in every octal digit), a digit every `pitch` bytes.
__device__ __forceinline__ void store_digits(const uint32_t (&digits)[16], unsigned char* out, int pitch) {
#pragma unroll
    for (int j = 0; j < kNativeDigits; ++j) {
        uint32_t word[2];
#pragma unroll
        for (int w = 0; w < 2; ++w) {
            uint32_t octal = 0;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int shift = 4 * i - 3 * j;
                const uint32_t moved = shift >= 0 ? digits[8 * w + i] << (shift & 31) : digits[8 * w + i] >> ((-shift) & 31);
                octal |= moved & ((j == kNativeDigits - 1 ? 15u : 7u) << (4 * i));
            }
            word[w] = e2m1_digits(octal, j == kNativeDigits - 1);
        }
        *reinterpret_cast<uint2*>(out + j * pitch) = make_uint2(word[0], word[1]);
    }
}

// The digits of what those of sixteen f16 that are below `on_grid` leave on the grid 1 / up, in multiples of 2^-23
// of it; one or two of them as a rule, so one after the other, all digits of a number at once.
__device__ __noinline__ void store_rest(uint4 lo, uint4 hi, uint32_t on_grid, float up, unsigned char* out, int pitch) {
    const uint32_t half[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
    uint32_t below = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        below |= ((half[i] & 0x7fffu) < on_grid ? 1u : 0u) << (2 * i);
        below |= (((half[i] >> 16) & 0x7fffu) < on_grid ? 2u : 0u) << (2 * i);
    }
    uint32_t word[kNativeDigits][2] = {};
#pragma unroll 1
    while (below != 0) {
        const int i = __ffs(below) - 1;
        below &= below - 1;
        uint32_t pair = half[0];
#pragma unroll
        for (int other = 1; other < 8; ++other) {
            pair = (i >> 1) == other ? half[other] : pair;
        }
        const float x = __half2float(__ushort_as_half(static_cast<unsigned short>((i & 1) ? pair >> 16 : pair))) * up;
        uint32_t octal = __float_as_uint(fmaf(x - rintf(x), 8388608.0f, kBinade)) + kToOctal;
        octal = (octal & 0xfffu) | (octal & 0xfff000u) << 4;  // three bits each -> a nibble each
        octal = (octal & 0x003f003fu) | (octal & 0x0fc00fc0u) << 2;
        octal = (octal & 0x07070707u) | (octal & 0x38383838u) << 1;
        const uint32_t codes = e2m1_digits(octal, false);
#pragma unroll
        for (int j = 0; j < kNativeDigits; ++j) {
            const uint32_t digit = ((codes >> (4 * j)) & 15u) << (4 * (i & 7));
            word[j][0] |= i < 8 ? digit : 0u;
            word[j][1] |= i < 8 ? 0u : digit;
        }
    }
#pragma unroll
    for (int j = 0; j < kNativeDigits; ++j) {
        *reinterpret_cast<uint2*>(out + j * pitch) = make_uint2(word[j][0], word[j][1]);
    }
}

// bf16 rows [batch][K] in and [batch][N] out.  A K split is a thread-block cluster that sums its slices, in
// slice order, through distributed shared memory: CTA s finishes the rows s, s + splits, ...
template <bool kSwiglu>
__global__ void __launch_bounds__(kNativeThreads, 1)
    nvfp4_native_kernel(const __grid_constant__ CUtensorMap map0, const __grid_constant__ CUtensorMap map1,
                        const __grid_constant__ CUtensorMap next_map0, const __grid_constant__ CUtensorMap next_map1,
                        const StreamKParams p) {
    extern __shared__ unsigned char smem_raw[];
    __shared__ NativeBarriers bars;
    unsigned char* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);

    pdl_launch_dependents();
    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const int cta = blockIdx.x;
    const int pair = cut_quotient(p.cut, cta);
    const int slice = cta - pair * p.splits;
    const int first_stage = cut_begin(p.cut, slice);
    const int num_stages = cut_begin(p.cut, slice + 1) - first_stage;
    const int group_blocks = p.in_features / 64;
    // activation rows padded to 2, 4 or 8
    const int rows_shift = p.batch <= 2 ? 1 : p.batch <= 4 ? 2 : 3;
    const int R = 1 << rows_shift;
    const int N = kNativeDigits * R;
    // digit tile [K / 32][N][16 bytes], its scale blocks, and the tile of the second eight digits
    const int x_slot_bytes = 2 * N * 128 + 2048;
    const int x_rest = N * 128 + 2048;
    const int x_slots = min(kNativeMaxXSlots, kNativeXBytes / x_slot_bytes);
    // a stage has 16 R blocks of 16 activations: one per lane of `team` warps
    const int team = R / 2;

    unsigned char* weight_ring = smem;  // [stage][tile][box | scales]
    unsigned char* x_ring = smem + kWeightStages * kTiles * kTileStageBytes;

    auto issue_stage = [&](int index) {
        const int slot = index % kWeightStages;
        const int stage = first_stage + index;
        int tile_row0[kTiles];
        int scale_tiles_present = 0;
#pragma unroll
        for (int t = 0; t < kTiles; ++t) {
            tile_row0[t] = kSwiglu ? pair * kTileRows : (pair * kTiles + t) * kTileRows;
            scale_tiles_present += tile_row0[t] < p.out_features ? 1 : 0;
        }
        mbar_arrive_expect_tx(&bars.w_full[slot], kTiles * kBoxBytes + scale_tiles_present * kScaleStageBytes);
#pragma unroll
        for (int t = 0; t < kTiles; ++t) {
            unsigned char* dst = weight_ring + (slot * kTiles + t) * kTileStageBytes;
            tma_box_g2s(dst, t == 1 ? &map1 : &map0, stage * kBoxRowBytes, tile_row0[t], &bars.w_full[slot]);
            if (tile_row0[t] < p.out_features) {
                bulk_g2s(dst + kBoxBytes,
                         p.scales[t] + (static_cast<size_t>(tile_row0[t] >> 7) * group_blocks + 4 * stage) * 512,
                         kScaleStageBytes, &bars.w_full[slot]);
            }
        }
    };
    // One stage before the CTA's barrier and the others after it, and nothing else in front of it that takes time
    // (nvfp4_streamk.cu): 34816 x 5120 at one row 18.3 -> 18.1 us, 5120 x 4096 6.29 -> 6.17.  The f16 kernel for
    // bf16 rows (nvfp4_umma.cu) gained nothing from it: 34816 x 5120 at 16 rows 21.3 / 21.3, pair at 32 rows 25.8 / 25.9.
    constexpr int early_stages = 1;
    if (threadIdx.x == 0) {
        for (int s = 0; s < kWeightStages; ++s) {
            mbar_init(&bars.w_full[s], 1);
            mbar_init(&bars.w_checked[s], 2);
            mbar_init(&bars.w_empty[s], 1);
        }
        mbar_fence_init();
        issue_stage(0);
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&bars.tmem_base)),
                     "r"(kTmemColumns)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    }
    if (threadIdx.x == 64) {
        for (int s = 0; s < kNativeMaxXSlots; ++s) {
            mbar_init(&bars.x_full[s], team);
            mbar_init(&bars.x_empty[s], 1);
            bars.rest[s] = 0;
        }
        bars.rest_used = 0;
        mbar_init(&bars.done, 1);
        bars.failed = 0;
        mbar_fence_init();
    }
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(&bars.tmem_base);
    // (by a thread that has time: whoever has to wait from here on looks at the flag)
    if (threadIdx.x == 64 && status_is_set(p.status)) {
        *reinterpret_cast<volatile int*>(&bars.failed) = 1;
    }
    int issued = early_stages;  // the producer's thread: stages asked for

    if (warp == 0) {
        // ---------------- weights ----------------
        bool ok = true;
        for (int index = early_stages; index < num_stages && ok; ++index) {
            const int slot = index % kWeightStages;
            ok = native_wait(&bars.w_empty[slot], ((index / kWeightStages) & 1) ^ 1, &bars, p.status);
            if (!ok) {
                break;
            }
            if (lane == 0) {
                issue_stage(index);
            }
            issued = index + 1;
            __syncwarp();
        }
        if (ok && p.next.valid && elect_one()) {
            prefetch_next_launch(p.next, next_map0, next_map1, cta, gridDim.x);
        }
    } else if (warp == 1) {
        // ---------------- tensor memory, scales, MMA ----------------
        // A and B e2m1 (1), scales e4m3, fp32 accumulators, M = 128
        const uint32_t idesc = (1u << 7) | (1u << 10) | (static_cast<uint32_t>(N >> 3) << 17) | (8u << 24);
        const uint32_t weight_base = smem_u32(weight_ring);
        const uint32_t x_base = smem_u32(x_ring);
        bool ok = true;
        int xs = 0;
        uint32_t x_parity = 0;
        uint32_t rest_started = 0;
        int index = 0;
        for (; index < num_stages; ++index) {
            const int slot = index % kWeightStages;
            ok = native_wait(&bars.w_checked[slot], (index / kWeightStages) & 1, &bars, p.status) &&
                 native_wait(&bars.x_full[xs], x_parity, &bars, p.status);
            if (!ok) {
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t rest = *reinterpret_cast<volatile uint32_t*>(&bars.rest[xs]);
            if (elect_one()) {
                const uint32_t scales = tmem_base + kNativeScaleColumn + (index & 1) * kNativeScaleColumns;
                const uint32_t x_tile = x_base + xs * x_slot_bytes;
                const uint32_t w_tile = weight_base + slot * kTiles * kTileStageBytes;
#pragma unroll
                for (int ks = 0; ks < 4; ++ks) {
#pragma unroll
                    for (int t = 0; t < kTiles; ++t) {
                        copy_scales(scales + 16 * t + 4 * ks,
                                    smem_descriptor(w_tile + t * kTileStageBytes + kBoxBytes + 512 * ks, 128, 128));
                    }
                    copy_scales(scales + 32 + 4 * ks, smem_descriptor(x_tile + N * 128 + 512 * ks, 128, 128));
                }
#pragma unroll
                for (int ks = 0; ks < 4; ++ks) {
                    const uint64_t b_desc = smem_descriptor(x_tile + ks * (2 * 16) * N, N * 16, 128);
#pragma unroll
                    for (int t = 0; t < kTiles; ++t) {
                        umma_nvfp4(tmem_base + t * kNativeAccumulator,
                                   swizzled_descriptor(w_tile + t * kTileStageBytes + 32 * ks), b_desc, idesc,
                                   scales + 16 * t + 4 * ks, scales + 32 + 4 * ks, (index > 0 || ks > 0) ? 1u : 0u);
                    }
                }
                if (rest != 0) {
                    uint32_t started = rest_started;
#pragma unroll 1
                    for (int ks = 0; ks < 4; ++ks) {
                        if (((rest >> (8 * ((ks * team) >> 2))) & 0xffu) == 0) {  // whose quarter of the stage it is
                            continue;
                        }
                        const uint64_t b_desc = smem_descriptor(x_tile + x_rest + ks * (2 * 16) * N, N * 16, 128);
#pragma unroll
                        for (int t = 0; t < kTiles; ++t) {
                            umma_nvfp4(tmem_base + t * kNativeAccumulator + kNativeRest,
                                       swizzled_descriptor(w_tile + t * kTileStageBytes + 32 * ks), b_desc, idesc,
                                       scales + 16 * t + 4 * ks, scales + 32 + 4 * ks, started);
                        }
                        started = 1;
                    }
                }
                umma_commit(&bars.w_empty[slot]);
                umma_commit(&bars.x_empty[xs]);
                if (index == num_stages - 1) {
                    umma_commit(&bars.done);
                }
            }
            __syncwarp();
            rest_started |= rest != 0 ? 1u : 0u;
            if (++xs == x_slots) {
                xs = 0;
                x_parity ^= 1;
            }
        }
        if (!ok && index > 0) {
            // the MMAs that were issued still read shared memory and write tensor memory: this warp waits for
            // the last of them (0.2 ms at most) before the CTA gives either back
            const long long start = clock64();
            while (!mbar_try_wait(&bars.w_empty[(index - 1) % kWeightStages], ((index - 1) / kWeightStages) & 1) &&
                   clock64() - start < 400000ll) {
            }
            __syncwarp();
        }
    } else if (warp < kNativeFirstWorker) {
        // ---------------- signs of the weight scales ----------------
        const int t = warp - 2;
        for (int index = 0; index < num_stages; ++index) {
            const int slot = index % kWeightStages;
            if (!native_wait(&bars.w_full[slot], (index / kWeightStages) & 1, &bars, p.status)) {
                break;
            }
            unsigned char* box = weight_ring + (slot * kTiles + t) * kTileStageBytes;
            uint4* blocks = reinterpret_cast<uint4*>(box + kBoxBytes);  // [K / 64][row % 32][row / 32][4]
            uint32_t signs = 0;
#pragma unroll
            for (int i = 0; i < kScaleStageBytes / 512; ++i) {
                const uint4 four = blocks[32 * i + lane];
                signs |= four.x | four.y | four.z | four.w;
            }
            if (__any_sync(0xffffffffu, (signs & 0x80808080u) != 0)) {
                for (int i = 0; i < kScaleStageBytes / 512; ++i) {
                    uint32_t* words = reinterpret_cast<uint32_t*>(blocks + 32 * i + lane);
                    for (int quarter = 0; quarter < 4; ++quarter) {
                        const uint32_t word = words[quarter];
                        const int row = quarter * 32 + lane;
                        for (int b = 0; b < 4; ++b) {
                            if ((word >> (8 * b + 7)) & 1u) {
                                // block 4 i + b of the row: eight bytes, half of a swizzled 16-byte piece
                                const int piece = (2 * i + (b >> 1)) ^ (row & 7);
                                uint2* codes = reinterpret_cast<uint2*>(box + row * kBoxRowBytes + piece * 16 + (b & 1) * 8);
                                *codes = make_uint2(codes->x ^ 0x88888888u, codes->y ^ 0x88888888u);
                            }
                        }
                        words[quarter] = word & 0x7f7f7f7fu;
                    }
                }
                fence_proxy_async();
            }
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(&bars.w_checked[slot]);
            }
        }
    } else {
        // ---------------- activations to digits ----------------
        const int e = warp - kNativeFirstWorker;
        pdl_wait();
        const int teams = kNativeWorkerWarps / team;
        const int task = (e % team) * 32 + lane;
        const int row = task & (R - 1);
        const int block = task >> rows_shift;  // of the stage's sixteen
        auto fetch = [&](int index, uint4& lo, uint4& hi) {
            const uint4* at = reinterpret_cast<const uint4*>(
                p.x_rows + static_cast<size_t>(min(row, p.batch - 1)) * p.in_features +
                (first_stage + index) * (kChunkK * kStageChunks) + 16 * block);
            lo = at[0];
            hi = at[1];
        };
        bool ok = true;
        bool rest_used = false;
        uint4 lo = make_uint4(0, 0, 0, 0), hi = lo;
        if (e / team < num_stages) {
            fetch(e / team, lo, hi);
        }
        for (int index = e / team; index < num_stages; index += teams) {
            uint32_t half[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
            if (index + teams < num_stages) {
                fetch(index + teams, lo, hi);
            }
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                half[i] = bf16x2_to_f16x2(half[i]);
            }
            uint32_t peak = 0;
            uint32_t least = 0x7fff7fffu;  // of the magnitudes that are not 0, less one, as signed halves from -32768
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const uint32_t magnitude = half[i] & 0x7fff7fffu;
                peak = __vmaxu2(peak, magnitude);
                least = __vmins2(least, magnitude + 0x7fff7fffu);
            }
            peak = max(peak & 0xffffu, peak >> 16);
            const int least_magnitude =
                min(static_cast<int>(static_cast<int16_t>(least & 0xffffu)), static_cast<int>(least) >> 16) + 0x8001;
            // the block's power of two: 2^(exponent - 14) is above every magnitude; below 2^-2 it stays, and
            // the last digit is then the grid of the smallest f16.  The scales end at 2^8 (2^7 of it is left
            // to the epilogue): the one binade above takes that scale, and its first digit may be 4.
            const int exponent = min(max(static_cast<int>(peak >> 10), 12), 29);
            // an e4m3 scale; NaN poisons the block (an infinity has become 65504 in the conversion)
            const uint32_t scale = peak >= 0x7c00u ? 0x7fu
                                   : exponent >= 15 ? static_cast<uint32_t>(exponent - 14) << 3
                                                    : 1u << (exponent - 12);
            const float up = __uint_as_float(static_cast<uint32_t>(163 - exponent) << 23);  // 2^(36 - exponent)
            // the smallest magnitude whose eight significant bits all lie on the grid of 2^(exponent - 36)
            const int on_grid = exponent <= 12 ? 0 : max(exponent - 14, 1) << 10;
            const bool again = __any_sync(0xffffffffu, least_magnitude < on_grid);
            rest_used |= again;
            // multiples of 2^(exponent - 36)
            uint32_t digits[16];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const float2 two = __half22float2(*reinterpret_cast<const __half2*>(&half[i]));
                digits[2 * i] = __float_as_uint(fmaf(two.x, up, kBinade)) + kToOctal;
                digits[2 * i + 1] = __float_as_uint(fmaf(two.y, up, kBinade)) + kToOctal;
                if (peak >= 0x7800u) {  // more than the binade holds
                    digits[2 * i] = static_cast<uint32_t>(__float2int_rn(two.x * up)) + 0x924924u;
                    digits[2 * i + 1] = static_cast<uint32_t>(__float2int_rn(two.y * up)) + 0x924924u;
                }
            }
            const int xs = index % x_slots;
            ok = native_wait(&bars.x_empty[xs], ((index / x_slots) & 1) ^ 1, &bars, p.status);
            if (!ok) {
                break;
            }
            unsigned char* tile = x_ring + xs * x_slot_bytes;
            unsigned char* out = tile + ((block >> 1) * N + row) * 16 + (block & 1) * 8;
            unsigned char* scale_out = tile + N * 128 + (block >> 2) * 512 + (block & 3);
#pragma unroll
            for (int j = 0; j < kNativeDigits; ++j) {
                const int n = j * R + row;
                scale_out[(n & 31) * 16 + (n >> 5) * 4] = static_cast<unsigned char>(scale);
            }
            store_digits(digits, out, R * 16);
            if (again) {
                store_rest(make_uint4(half[0], half[1], half[2], half[3]), make_uint4(half[4], half[5], half[6], half[7]),
                           static_cast<uint32_t>(on_grid), up, out + x_rest, R * 16);
            }
            if (lane == 0) {
                reinterpret_cast<volatile uint8_t*>(&bars.rest[xs])[e % team] = again ? 1 : 0;
            }
            fence_proxy_async();
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(&bars.x_full[xs]);
            }
        }
        if (rest_used && lane == 0) {
            *reinterpret_cast<volatile int*>(&bars.rest_used) = 1;
        }
        __syncwarp();
        asm volatile("bar.sync 1, %0;" ::"n"(kNativeWorkerWarps * 32) : "memory");
        // ---------------- epilogue ----------------
        // Warp e: output rows 32 (e % 4) .. + 31 of both tiles, activation rows (e / 4) R / 2 .. .
        ok = native_wait(&bars.done, 0, &bars, p.status) &&
             __all_sync(0xffffffffu, *reinterpret_cast<volatile int*>(&bars.failed) == 0);
        if (ok) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const int quarter = e & 3;
            const int first_token = (e >> 2) * (R / 2);
            const uint32_t address = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + first_token;
            constexpr int kTokens = kNativeRows / 2;
            float v0[kTokens], v1[kTokens];
#pragma unroll
            for (int i = 0; i < kTokens; ++i) {
                v0[i] = v1[i] = 0.0f;
            }
            const auto add_digits = [&](uint32_t columns, float weight) {  // `weight` of the lowest digit
#pragma unroll
                for (int first = 0; first < kNativeDigits; first += 4) {
                    uint32_t r0[4][8], r1[4][8];  // (the columns behind this warp's rows are other rows and digits)
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        tmem_load8_issue(columns + (first + j) * R, r0[j]);
                        tmem_load8_issue(columns + kNativeAccumulator + (first + j) * R, r1[j]);
                    }
                    tmem_load_wait();
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
#pragma unroll
                        for (int i = 0; i < kTokens; ++i) {
                            v0[i] = fmaf(__uint_as_float(r0[j][i]), weight, v0[i]);
                            v1[i] = fmaf(__uint_as_float(r1[j][i]), weight, v1[i]);
                        }
                        weight *= 8.0f;
                    }
                }
            };
            constexpr float kLowest = 128.0f / 2097152.0f;  // 2^7 8^-7
            if (*reinterpret_cast<volatile int*>(&bars.rest_used) != 0) {
                add_digits(address + kNativeRest, kLowest / 8388608.0f);
            }
            add_digits(address, kLowest);
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            const int tokens = min(p.batch - first_token, R / 2);
            if (p.splits > 1) {
                // every stage has been consumed: the weight ring is free to park the sums in
                float* park = reinterpret_cast<float*>(weight_ring) + quarter * 32 + lane;
#pragma unroll
                for (int i = 0; i < kTokens; ++i) {
                    if (i < tokens) {
                        park[(first_token + i) * kTileRows] = v0[i];
                        park[(kNativeRows + first_token + i) * kTileRows] = v1[i];
                    }
                }
            } else {
                const int row0 = (kSwiglu ? pair * kTileRows : pair * kTiles * kTileRows) + quarter * 32 + lane;
#pragma unroll
                for (int i = 0; i < kTokens; ++i) {
#pragma unroll
                    for (int t = 0; t < (kSwiglu ? 1 : kTiles); ++t) {
                        const int out_row = row0 + t * kTileRows;
                        if (i < tokens && out_row < p.out_features) {
                            float value = (t == 0 ? v0[i] : v1[i]) * p.inverse_scale[0];
                            if (kSwiglu) {
                                value = value / (1.0f + __expf(-value)) * (v1[i] * p.inverse_scale[1]);
                            }
                            p.y[static_cast<size_t>(first_token + i) * p.out_features + out_row] =
                                __float2bfloat16(value);
                        }
                    }
                }
            }
        }
    }

    if (p.splits > 1) {
        native_cluster_sync();
        const int worker = static_cast<int>(threadIdx.x) - kNativeFirstWorker * 32;
        const int t = worker >> 7;
        const int out_row = kSwiglu ? pair * kTileRows + (worker & 127)
                                    : (pair * kTiles + t) * kTileRows + (worker & 127);
        if (worker >= 0 && (!kSwiglu || t == 0) && out_row < p.out_features) {
            uint32_t gave_up = 0;  // a CTA that did has no sums: nobody of its cluster stores
#pragma unroll
            for (int r = 0; r < 8; ++r) {
                gave_up |= r < p.splits ? native_peer_word(&bars.failed, r) : 0u;
            }
            for (int token = slice; token < p.batch; token += p.splits) {
                const float* park =
                    reinterpret_cast<const float*>(weight_ring) + (t * kNativeRows + token) * kTileRows + (worker & 127);
                float part[8], gate_up[8];
#pragma unroll
                for (int r = 0; r < 8; ++r) {  // all slices in flight at once
                    part[r] = r < p.splits ? native_peer_float(park, r) : 0.0f;
                    gate_up[r] = kSwiglu && r < p.splits ? native_peer_float(park + kNativeRows * kTileRows, r) : 0.0f;
                }
                float value = 0.0f, up = 0.0f;
#pragma unroll
                for (int r = 0; r < 8; ++r) {
                    value += part[r];
                    up += gate_up[r];
                }
                value *= p.inverse_scale[0];
                if (kSwiglu) {
                    value = value / (1.0f + __expf(-value)) * (up * p.inverse_scale[1]);
                }
                if (gave_up == 0) {
                    p.y[static_cast<size_t>(token) * p.out_features + out_row] = __float2bfloat16(value);
                }
            }
        }
        native_cluster_sync();  // nobody leaves while a peer may still read its shared memory
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (*reinterpret_cast<volatile int*>(&bars.failed) != 0 && threadIdx.x == 0) {
        // stages asked for may still be landing in this CTA's shared memory (a wait of 0.2 ms per slot)
        for (int index = max(0, issued - kWeightStages); index < issued; ++index) {
            const long long start = clock64();
            while (!mbar_try_wait(&bars.w_full[index % kWeightStages], (index / kWeightStages) & 1) &&
                   clock64() - start < 400000ll) {
            }
        }
    }
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kTmemColumns) : "memory");
    }
}

}  // namespace
}  // namespace qwc
