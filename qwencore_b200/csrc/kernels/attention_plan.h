// The split plan of the packed attention kernel: which piece of which row a chunk of work is.  Plain arithmetic, the
// same on the device and on the host, where it can be walked through at sizes that no cache holds.

#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define QWC_PLAN_FUNCTION __host__ __device__ __forceinline__
#else
#define QWC_PLAN_FUNCTION inline
#endif

namespace qwc {
namespace {

constexpr int kUnitTokens = 16;
constexpr int kStageUnits = 8;
constexpr int kPlanKvHeads = 4;
constexpr int kPlanMinPadding = 4;        // units a task costs beyond its tokens
constexpr int kPlanPaddingDivisor = 64;   // padding = share / this at least: bounds the tasks of one chunk
constexpr int kMaxPairsPerSm = 38;        // (256 rows on 27 SMs)
constexpr int kMaxListTasks = kMaxPairsPerSm + kPlanPaddingDivisor + 4;  // tasks of one chunk (plan_fits)
constexpr int kChunksPerSm = 4;           // one large chunk and three small ones
constexpr int kDynamicShare = 192;        // units per SM from which on the line is cut into chunks of two sizes ...
constexpr int kThreeSmallShare = 480;     // ... with three small ones instead of two
constexpr int kPlanRows = 256;            // rows whose prefix fits the shared-memory table

// The split plan.
//
// The (row, kv head) pairs are laid end to end, row-major, on a line of units; a pair takes
// max(units, 1) + padding positions (the padding stands for what a task costs beyond its tokens).
// The line is cut into chunks, and a task is the piece of one pair inside one chunk, partial number
// c - (first chunk that touches the pair); a pair without context is one empty piece.  The last piece of a pair says
// so in the sign of its sum: the merge kernel needs no plan.
//   * One equal chunk per SM, up to kDynamicShare units.  Beyond that one large chunk (seven tenths of an SM's share)
//     and two or, from kThreeSmallShare on, three small ones: a CTA starts with a large chunk and, once it has
//     asked for its last bytes, takes the next chunk that nobody has.  The SMs do not get the same share of the
//     memory's bandwidth (40 to 56 GB/s each, others every time): with equal chunks of 350 units the CTAs' ends
//     lay 53 to 72 us after their first copies.  Measured (us, equal chunks / two small / three small / six small):
//     share 350 (32 rows, log-uniform to 32768) 79.9 / 77.2 / 78.6 / 83.4, 330 76.0 / 71.8 / 72.8, 612 (20 rows,
//     8192 to 32768) 128.5 / 123.0 / 121.1 / 126.1, 230 (32 x 4096) 56.3 / 55.2 / 58.2; at 166 (three rows of
//     32768, forced) 42.8 / - / 52.1.
//   * padding >= share / kPlanPaddingDivisor, so that a chunk never holds more than kPlanPaddingDivisor + 4 tasks and
//     one per pair and SM (what the padding itself adds to a share);
//   * every chunk >= capacity / (partitions - 1): a row never has more pieces than the workspace has slots;
//   * every chunk is a whole number of stages.
// Position: uint32_t, unless a launch could have chunks that end beyond that (PlanShape::wide).
template <typename Position>
struct SplitPlan {
    Position large, small;
    Position line;
    int padding;
};

template <typename Position>
QWC_PLAN_FUNCTION SplitPlan<Position> make_split_plan(Position total_row_units, int rows, int smallest_chunk,
                                                      int ctas) {
    // (shares in floating point, rounded up by more than the arithmetic can be off)
    const float per_cta = 1.00001f / static_cast<float>(ctas);
    const Position smallest = static_cast<Position>(smallest_chunk);
    Position share = static_cast<Position>(static_cast<float>(total_row_units) * kPlanKvHeads * per_cta) + 1;
    share = share > smallest ? share : smallest;
    SplitPlan<Position> plan;
    plan.padding = static_cast<int>(share / kPlanPaddingDivisor) + 1;
    plan.padding = plan.padding > kPlanMinPadding ? plan.padding : kPlanMinPadding;
    plan.line = (total_row_units + static_cast<Position>(rows) * plan.padding) * kPlanKvHeads;
    share = static_cast<Position>(static_cast<float>(plan.line) * per_cta) + 1;
    const bool dynamic = share >= kDynamicShare;
    const Position tenth = share / 10;
    plan.small = !dynamic ? share : share >= kThreeSmallShare ? tenth : tenth + tenth / 2;
    plan.large = !dynamic ? share : share - (share >= kThreeSmallShare ? 3 : 2) * plan.small;
    plan.large = ((plan.large > smallest ? plan.large : smallest) + kStageUnits - 1) / kStageUnits * kStageUnits;
    plan.small = ((plan.small > smallest ? plan.small : smallest) + kStageUnits - 1) / kStageUnits * kStageUnits;
    return plan;
}

// The chunk that holds a position of the line ...
template <typename Position>
QWC_PLAN_FUNCTION int chunk_of(const SplitPlan<Position>& plan, Position position, int ctas) {
    const Position small_begin = plan.large * ctas;
    return position < small_begin ? static_cast<int>(position / plan.large)
                                  : ctas + static_cast<int>((position - small_begin) / plan.small);
}

// ... and where a chunk begins.
template <typename Position>
QWC_PLAN_FUNCTION Position chunk_begin(const SplitPlan<Position>& plan, int chunk, int ctas) {
    return chunk < ctas ? plan.large * chunk : plan.large * ctas + plan.small * (chunk - ctas);
}

// first position of pair (row, kv head); units_before = units of the rows before it
template <typename Position>
QWC_PLAN_FUNCTION Position pair_position(const SplitPlan<Position>& plan, int row, int kv_head, Position units_before,
                                         Position row_units) {
    return (units_before + static_cast<Position>(row) * plan.padding) * kPlanKvHeads +
           static_cast<Position>(kv_head) * (row_units + plan.padding);
}

// Whether a pair at [start, start + occupied) has a piece inside the chunk [low, high), and the piece.
struct PlanPiece {
    int begin, end;  // its units, counted from the pair's first (a row without context: end 1)
    int part;
    bool last;  // no piece of the pair after this one
};

template <typename Position>
QWC_PLAN_FUNCTION bool piece_inside(Position start, Position occupied, Position low, Position high) {
    return start < high && start + occupied > low;
}

template <typename Position>
QWC_PLAN_FUNCTION PlanPiece piece_of_pair(const SplitPlan<Position>& plan, Position start, Position occupied, int chunk,
                                          Position low, Position high, int ctas) {
    PlanPiece piece;
    piece.begin = static_cast<int>(low > start ? low - start : 0);
    piece.end = static_cast<int>(high - start < occupied ? high - start : occupied);
    piece.part = start < low ? chunk - chunk_of(plan, start, ctas) : 0;
    piece.last = piece.end == static_cast<int>(occupied);
    return piece;
}

// A context longer than the block table can describe is cut at the table's capacity.
QWC_PLAN_FUNCTION int units_of_context(uint32_t context, int capacity_units) {
    const uint32_t units = (context + kUnitTokens - 1) / kUnitTokens;
    return static_cast<int>(units < static_cast<uint32_t>(capacity_units) ? units : capacity_units);
}

// Units a row occupies on the plan's line: a row without context still gets one task (it stores zeros).
QWC_PLAN_FUNCTION int plan_units(int units) { return units > 0 ? units : 1; }

// Whether a list holds the tasks of every chunk (undivided rows: one per pair and SM).
inline bool plan_fits(int rows, int ctas) { return (rows * kPlanKvHeads + ctas - 1) / ctas <= kMaxPairsPerSm; }

// What the launcher decides about the plan before it knows any context: a bound over all contexts that the block
// tables can describe.
struct PlanShape {
    int smallest_chunk;   // units; a row never has more pieces than `partitions`
    bool wide;            // positions need more than 32 bits
    bool may_be_dynamic;  // chunks may have two sizes: the grid has kChunksPerSm CTAs per SM
};

inline PlanShape plan_shape(int rows, int max_blocks, int page_size, int partitions, int ctas) {
    // (a context is a 32-bit number of tokens, whatever the tables could describe)
    const long long described = static_cast<long long>(max_blocks) * (page_size / kUnitTokens);
    const long long capacity = described < (1ll << 28) ? described : (1ll << 28);
    const long long smallest = (capacity + partitions - 2) / (partitions - 1);
    // make_split_plan step by step with every row at the capacity: no term of it shrinks when a context grows, but for
    // the line between one size of chunks and two.  (A share is rounded up by less than 2^-16 of itself.)
    const auto share_of = [ctas](long long units) { return (units + (units >> 16)) / ctas + 2; };
    const long long share = share_of(capacity * rows * kPlanKvHeads);
    const long long padding = (share > smallest ? share : smallest) / kPlanPaddingDivisor + 1 + kPlanMinPadding;
    const long long padded_share = share_of((capacity + padding) * rows * kPlanKvHeads);
    const long long chunk = (padded_share > smallest ? padded_share : smallest) + kStageUnits;
    PlanShape shape;
    shape.smallest_chunk = static_cast<int>(smallest);
    shape.wide = chunk * kChunksPerSm * ctas >= (1ll << 32);  // where the last chunk ends, used or not
    shape.may_be_dynamic = padded_share >= kDynamicShare;
    return shape;
}

}  // namespace
}  // namespace qwc
