// The split plan of the packed attention kernel, walked through on the host as the plan warps of all CTAs would, with
// the position type and the grid that the launcher chooses.  Exit code 0: every unit of every row is in exactly one
// piece, every piece has a slot of the workspace and is the work of a chunk that the grid has, no list overflows.

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <random>
#include <vector>

#include "attention_plan.h"

using namespace qwc;

namespace {

struct Call {
    int rows, max_blocks, page_size, partitions, ctas;
    std::vector<uint32_t> contexts;
};

bool fail(const Call& c, const char* what, long long a, long long b) {
    std::printf("%s (%lld, %lld): rows %d blocks %d page %d partitions %d ctas %d\n", what, a, b, c.rows, c.max_blocks,
                c.page_size, c.partitions, c.ctas);
    return false;
}

template <typename Position>
bool walk(const Call& c, const PlanShape& shape) {
    const int grid = shape.may_be_dynamic ? kChunksPerSm * c.ctas : c.ctas;
    const int capacity = static_cast<int>(
        std::min<long long>(static_cast<long long>(c.max_blocks) * (c.page_size / kUnitTokens), 1ll << 28));
    std::vector<Position> first(c.rows + 1, 0);
    for (int r = 0; r < c.rows; ++r) {
        first[r + 1] = first[r] + plan_units(units_of_context(c.contexts[r], capacity));
    }
    const auto plan = make_split_plan<Position>(first[c.rows], c.rows, shape.smallest_chunk, c.ctas);
    std::vector<long long> covered(c.rows * kPlanKvHeads, 0);
    std::vector<int> parts(c.rows * kPlanKvHeads, 0);
    for (int chunk = 0; chunk < grid; ++chunk) {
        const Position low = chunk_begin(plan, chunk, c.ctas), high = chunk_begin(plan, chunk + 1, c.ctas);
        if (chunk >= c.ctas && low >= plan.line) {
            continue;  // claimed and dropped
        }
        int tasks = 0;
        for (int pair = 0; pair < c.rows * kPlanKvHeads; ++pair) {
            const int r = pair / kPlanKvHeads;
            const Position occupied = first[r + 1] - first[r];
            const Position start = pair_position(plan, r, pair % kPlanKvHeads, first[r], occupied);
            if (start >= high) {
                break;
            }
            if (!piece_inside(start, occupied, low, high)) {
                continue;
            }
            const PlanPiece piece = piece_of_pair(plan, start, occupied, chunk, low, high, c.ctas);
            if (piece.part != parts[pair] || piece.part >= c.partitions) {
                return fail(c, "slot of a piece", piece.part, parts[pair]);
            }
            if (piece.begin != covered[pair] || piece.end <= piece.begin) {
                return fail(c, "units of a piece", piece.begin, covered[pair]);
            }
            covered[pair] = piece.end;
            ++parts[pair];
            if (piece.last != (static_cast<Position>(piece.end) == occupied)) {
                return fail(c, "mark of the last piece", piece.end, piece.last);
            }
            ++tasks;
        }
        if (tasks > kMaxListTasks) {
            return fail(c, "tasks of a chunk", tasks, kMaxListTasks);
        }
    }
    for (int pair = 0; pair < c.rows * kPlanKvHeads; ++pair) {
        if (covered[pair] != static_cast<long long>(first[pair / kPlanKvHeads + 1] - first[pair / kPlanKvHeads])) {
            return fail(c, "units without a chunk", pair, covered[pair]);
        }
    }
    return true;
}

bool check(const Call& c) {
    if (!plan_fits(c.rows, c.ctas)) {
        return fail(c, "refused", c.rows, c.ctas);
    }
    const PlanShape shape = plan_shape(c.rows, c.max_blocks, c.page_size, c.partitions, c.ctas);
    return shape.wide ? walk<unsigned long long>(c, shape) : walk<uint32_t>(c, shape);
}

}  // namespace

int main() {
    std::mt19937_64 rng(1);
    const auto below = [&rng](double limit) { return std::uniform_real_distribution<double>(0.0, limit)(rng); };
    long long calls = 0, wide = 0, dynamic = 0;
    const int cta_counts[] = {148, 132, 74, 37, 27, 8};
    for (int round = 0; round < 6000; ++round) {
        Call c;
        c.ctas = cta_counts[round % 6];
        c.page_size = rng() % 2 ? 16 : 64;
        // up to 38 (row, kv head) pairs per SM
        const int most_rows = std::min(kPlanRows, 38 * c.ctas / kPlanKvHeads);
        c.rows = round % 7 == 0 ? most_rows : 1 + static_cast<int>(std::exp2(below(8.0)) - 1) % most_rows;
        c.max_blocks = static_cast<int>(std::exp2(below(28.0)));
        c.partitions = 2 + static_cast<int>(std::exp2(below(12.0)) - 1);
        const int kind = static_cast<int>(rng() % 4);
        const double longest = std::min<double>(4294967295.0, static_cast<double>(c.max_blocks) * c.page_size);
        for (int r = 0; r < c.rows; ++r) {
            // every row full (or past the table), one long among short ones, log-uniform, none
            const double tokens = kind == 0 ? longest
                                  : kind == 1 ? (r == c.rows / 2 ? longest : below(100.0))
                                  : kind == 2 ? std::exp2(below(std::log2(longest + 1.0))) - 1.0
                                              : (rng() % 3 ? 0.0 : below(longest));
            c.contexts.push_back(static_cast<uint32_t>(tokens));
        }
        if (!check(c)) {
            return 1;
        }
        const PlanShape shape = plan_shape(c.rows, c.max_blocks, c.page_size, c.partitions, c.ctas);
        ++calls;
        wide += shape.wide;
        dynamic += shape.may_be_dynamic;
    }
    // a line just below 2^31 whose smallest chunk makes the chunks end past 2^32
    if (!check({60, 1800000, 64, 2, 148, std::vector<uint32_t>(60, 115200000u)})) {
        return 1;
    }
    // short rows, whose padding brings the share of an SM over the line between one size of chunks and two
    if (!check({196, 3, 16, 8, 28, std::vector<uint32_t>(196, 48u)})) {
        return 1;
    }
    // contexts at the largest numbers of tokens that a launch can be given
    if (!check({32, 1 << 28, 16, 2, 148, std::vector<uint32_t>(32, 0xfffffff0u)})) {
        return 1;
    }
    std::printf("ok calls=%lld wide=%lld dynamic=%lld\n", calls, wide, dynamic);
    return 0;
}
