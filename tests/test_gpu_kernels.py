"""GPU parity: every kernel through the C ABI against the CPU oracle on seeded inputs.

Tolerances: floating-point outputs must satisfy max|gpu - oracle| <= 1e-2 * RMS(oracle)
(the bound the north star states); indexing, page tables, slot packing and the int8
requantiser are compared bit for bit.  Where the reference has its own test for a case,
its name and tolerance are cited and also applied.
"""

import numpy as np
import pytest

from oracle import oracle
from qwencore_b200 import synth

pytestmark = pytest.mark.gpu

RMS_BOUND = 1.0e-2


def dev(torch, array):
    return torch.from_numpy(np.ascontiguousarray(array)).cuda()


def host(tensor):
    return tensor.detach().cpu().numpy()


def bf16_out(torch, *shape):
    return dev(torch, np.zeros(shape, dtype=np.uint16))


def u32_out(torch, *shape, fill=0):
    return dev(torch, np.full(shape, fill, dtype=np.uint32))


# (comparison, elements that needed the bf16 grid term on top of 1e-2 * RMS, elements compared)
GRID_TERM_USE = []


def assert_rms_close(got, want, what, bound=RMS_BOUND, bf16_grid=True):
    """max|got - want| <= bound * RMS(want).  A bf16 output cannot meet that bound by itself
    beyond 2.6 RMS (its grid step there exceeds 1e-2 RMS), so for bf16 outputs one grid step
    of the expected value (at most 2^-7 relative) is allowed on top."""
    got = np.asarray(got, dtype=np.float64)
    want = np.asarray(want, dtype=np.float64)
    rms = np.sqrt(np.mean(want ** 2))
    assert np.isfinite(got).all(), f"{what}: non-finite output"
    allowed = bound * rms + (2.0 ** -7 * np.abs(want) if bf16_grid else 0.0)
    if bf16_grid:  # how many elements the plain bound alone would have failed: printed with the test summary
        GRID_TERM_USE.append((what, int(np.count_nonzero(np.abs(got - want) > bound * rms)), int(got.size)))
    excess = np.abs(got - want) - allowed
    worst = np.unravel_index(np.argmax(excess), excess.shape)
    assert excess[worst] <= 0, (f"{what}: |{got[worst]:.6g} - {want[worst]:.6g}| exceeds {bound} * rms "
                                f"{rms:.4g} at {worst}")


@pytest.fixture(scope="module")
def ops(cuda, built_library):
    from qwencore_b200 import abi, ops as module

    yield module
    assert abi.lib.qwc_device_status() == 0, "a bounded device wait gave up during the tests"


class LcgRng:
    """The generator of the reference's GEMV test (crates/qwc-cuda/tests/nvfp4.rs:7-21)."""

    def __init__(self, seed):
        self.state = seed

    def next_u8(self):
        self.state = (self.state * 6364136223846793005 + 1442695040888963407) & 0xFFFFFFFFFFFFFFFF
        return self.state >> 56

    def next_f32(self):
        return np.float32(np.float32(self.next_u8()) / np.float32(255.0) * np.float32(2.0) - np.float32(1.0))


# ---------------------------------------------------------------------------------------
# NVFP4 W4A16
# ---------------------------------------------------------------------------------------

def run_gemv(torch, ops, packed, scales, swizzled, global_scale, x_bits, out_features, in_features, batch):
    linear = ops.Linear(dev(torch, packed), dev(torch, swizzled), global_scale, out_features, in_features)
    out = bf16_out(torch, batch, out_features)
    linear.forward_w4a16(dev(torch, x_bits), out, batch)
    torch.cuda.synchronize()
    return synth.bf16_value(host(out)), linear


def test_w4a16_matches_cpu_for_all_supported_batches(cuda, ops):
    """crates/qwc-cuda/tests/nvfp4.rs:23-111 (OUT = 37 checks a ragged last tile), extended to 32 rows."""
    torch = cuda
    OUT, IN = 37, 512
    rng = LcgRng(0x4A165090)
    packed = np.array([rng.next_u8() for _ in range(OUT * IN // 2)], dtype=np.uint8).reshape(OUT, IN // 2)
    up_packed = np.array([rng.next_u8() for _ in range(OUT * IN // 2)], dtype=np.uint8).reshape(OUT, IN // 2)
    codes = [0x30, 0x38, 0x3C, 0x40]
    scales = np.array([codes[i % 4] for i in range(OUT * IN // 16)], dtype=np.uint8).reshape(OUT, IN // 16)
    swizzled = synth.swizzle_block_scales(scales, OUT, IN)
    for batch in [1, 2, 3, 4, 7, 8, 9, 16, 17, 31, 32]:
        x = synth.bf16_bits(np.array([rng.next_f32() for _ in range(batch * IN)], dtype=np.float32).reshape(batch, IN))
        want = oracle.gemv_w4a16(packed, scales, 8.0, x, OUT, IN, batch)
        got, gate = run_gemv(torch, ops, packed, scales, swizzled, 8.0, x, OUT, IN, batch)
        tolerance = 0.035 + np.abs(want) * 0.012  # tests/nvfp4.rs:68
        assert np.all(np.abs(got - want) <= tolerance), f"batch {batch}"

        want_up = oracle.gemv_w4a16(up_packed, scales, 4.0, x, OUT, IN, batch)
        want_fused = oracle.swiglu_combine(want, want_up)
        up = ops.Linear(dev(torch, up_packed), dev(torch, swizzled), 4.0, OUT, IN)
        fused = bf16_out(torch, batch, OUT)
        ops.swiglu_w4a16(gate, up, dev(torch, x), fused, batch)
        torch.cuda.synchronize()
        got_fused = synth.bf16_value(host(fused))
        tolerance = 0.075 + np.abs(want_fused) * 0.025  # tests/nvfp4.rs:103
        assert np.all(np.abs(got_fused - want_fused) <= tolerance), f"fused batch {batch}"


@pytest.mark.parametrize("out_features,in_features,batches", [
    (34816, 5120, [1, 32]),      # benchmark config 0 shape (fused gate_up) and the c=32 case
    (12352, 5120, [5, 16]),      # mixer in-proj of the 32-value-head model: 96.5 row blocks
    (5120, 17408, [1, 8, 32]),   # down: narrow output, K split across a cluster
    (5120, 4096, [2, 24]),       # la_out
    (1024, 5120, [1, 12]),       # k / v projections
])
def test_w4a16_model_shapes_up_to_32_rows_oracle_generalisation_beyond_reference_batch_8(cuda, ops, out_features,
                                                                                          in_features, batches):
    torch = cuda
    packed, scales, swizzled = synth.nvfp4_matrix(0, f"w{out_features}x{in_features}", out_features, in_features)
    for batch in batches:
        x = synth.normal_bf16(0, f"x{batch}", (batch, in_features))
        want = oracle.gemv_w4a16(packed, scales, 1.0, x, out_features, in_features, batch)
        got, _ = run_gemv(torch, ops, packed, scales, swizzled, 1.0, x, out_features, in_features, batch)
        assert_rms_close(got, oracle.bf16_round(want), f"gemv {out_features}x{in_features} b{batch}")


def test_prefetch_next_hint_changes_no_result_and_rejects_bad_arguments(cuda, ops):
    """qwc_nvfp4_prefetch_next only moves lines into L2: a hinted launch stores the same bytes."""
    torch = cuda
    from qwencore_b200 import abi
    N, K, batch = 5120, 6144, 32
    packed, scales, swizzled = synth.nvfp4_matrix(3, "hinted", N, K)
    other_p, _, other_sw = synth.nvfp4_matrix(3, "after", 12352, 5120)
    up_p, _, up_sw = synth.nvfp4_matrix(3, "after_up", 12352, 5120)
    x = dev(torch, synth.normal_bf16(3, "x", (batch, K)))
    linear = ops.Linear(dev(torch, packed), dev(torch, swizzled), 1.0, N, K)
    after = ops.Linear(dev(torch, other_p), dev(torch, other_sw), 1.0, 12352, 5120)
    after_up = ops.Linear(dev(torch, up_p), dev(torch, up_sw), 1.0, 12352, 5120)
    plain = bf16_out(torch, batch, N)
    linear.forward_w4a16(x, plain, batch)
    for second in (None, after_up):
        hinted = bf16_out(torch, batch, N)
        ops.prefetch_next(after, second)
        linear.forward_w4a16(x, hinted, batch)
        torch.cuda.synchronize()
        assert np.array_equal(host(hinted), host(plain))
    table = torch.zeros((4096, 5120), dtype=torch.uint8, device="cuda")
    assert abi.lib.qwc_nvfp4_prefetch_next(table.data_ptr(), None, None, None, 4096, 5120, 2) == 0
    hinted = bf16_out(torch, batch, N)
    linear.forward_w4a16(x, hinted, batch)
    torch.cuda.synchronize()
    assert np.array_equal(host(hinted), host(plain))
    invalid = 1  # cudaErrorInvalidValue
    good = (after.packed.data_ptr(), after.scales.data_ptr())
    assert abi.lib.qwc_nvfp4_prefetch_next(None, good[1], None, None, 12352, 5120, 0) == invalid
    assert abi.lib.qwc_nvfp4_prefetch_next(good[0], None, None, None, 12352, 5120, 0) == invalid
    assert abi.lib.qwc_nvfp4_prefetch_next(good[0], good[1], None, None, 12352, 5120, 1) == invalid
    assert abi.lib.qwc_nvfp4_prefetch_next(good[0], good[1], None, None, 12352, 5000, 0) == invalid
    assert abi.lib.qwc_nvfp4_prefetch_next(good[0], good[1], None, None, 0, 5120, 0) == invalid
    assert abi.lib.qwc_nvfp4_prefetch_next(good[0], good[1], None, None, 12352, 5120, 5) == invalid
    assert abi.lib.qwc_nvfp4_prefetch_next(good[0] + 8, good[1], None, None, 12352, 5120, 0) == invalid
    assert abi.lib.qwc_device_status() == 0


@pytest.mark.parametrize("batch", [1, 6, 13, 32])
def test_swiglu_w4a16_mlp_shape(cuda, ops, batch):
    torch = cuda
    N, K = 17408, 5120
    gate_p, gate_s, gate_sw = synth.nvfp4_matrix(1, "gate", N, K)
    up_p, up_s, up_sw = synth.nvfp4_matrix(1, "up", N, K)
    x = synth.normal_bf16(1, f"x{batch}", (batch, K), std=0.25)
    want = oracle.swiglu_combine(oracle.gemv_w4a16(gate_p, gate_s, 2.0, x, N, K, batch),
                                 oracle.gemv_w4a16(up_p, up_s, 4.0, x, N, K, batch))
    gate = ops.Linear(dev(torch, gate_p), dev(torch, gate_sw), 2.0, N, K)
    up = ops.Linear(dev(torch, up_p), dev(torch, up_sw), 4.0, N, K)
    out = bf16_out(torch, batch, N)
    ops.swiglu_w4a16(gate, up, dev(torch, x), out, batch)
    torch.cuda.synchronize()
    assert_rms_close(synth.bf16_value(host(out)), oracle.bf16_round(want), f"swiglu b{batch}")


def test_w4a16_rejects_bad_arguments(cuda, ops):
    from qwencore_b200 import abi

    lib = abi.lib
    buffer = cuda.zeros(4096, dtype=cuda.uint8, device="cuda").data_ptr()
    assert lib.qwc_nvfp4_w4a16(0, buffer, buffer, buffer, 16, 256, 1, 1.0, 0) == abi.CUDA_ERROR_INVALID_VALUE
    assert lib.qwc_nvfp4_w4a16(buffer, buffer, buffer, buffer, 16, 128, 1, 1.0, 0) == abi.CUDA_ERROR_INVALID_VALUE
    assert lib.qwc_nvfp4_w4a16(buffer, buffer, buffer, buffer, 16, 256, 33, 1.0, 0) == abi.CUDA_ERROR_INVALID_VALUE
    assert lib.qwc_nvfp4_w4a16(buffer, buffer, buffer, buffer, 16, 256, 1, 0.0, 0) == abi.CUDA_ERROR_INVALID_VALUE


# ---------------------------------------------------------------------------------------
# Packed paged attention
# ---------------------------------------------------------------------------------------

def run_attention(torch, ops, case, page_size, partitions, batch=None):
    batch = batch or case["contexts"].size
    out = bf16_out(torch, batch, 24, 256)
    workspace = None
    if partitions > 1:
        workspace = torch.zeros(ops.packed_workspace_bytes(batch, partitions), dtype=torch.uint8, device="cuda")
    gate = None if case["gate_projection"] is None else dev(torch, case["gate_projection"])
    ks = None if case["k_scale"] is None else dev(torch, case["k_scale"])
    vs = None if case["v_scale"] is None else dev(torch, case["v_scale"])
    ops.gated_packed(dev(torch, case["query"]), gate, dev(torch, case["key_cache"]), dev(torch, case["value_cache"]),
                     dev(torch, case["block_tables"]), dev(torch, case["contexts"]), case["max_blocks"], out, batch, 0,
                     partitions, workspace, page_size, ks, vs)
    torch.cuda.synchronize()
    return synth.bf16_value(host(out))


def attention_oracle(case, page_size):
    return oracle.paged_attention_fp8(case["query"], case["gate_projection"], case["key_cache"], case["value_cache"],
                                      case["block_tables"], case["contexts"], case["max_blocks"],
                                      batch=case["contexts"].size, page_size=page_size, k_scale=case["k_scale"],
                                      v_scale=case["v_scale"])


def check_attention(got, want, what):
    # reference tolerance (crates/qwc-cuda/tests/paged_attention.rs:115,888) and the RMS bound
    assert np.all(np.abs(got - want) <= 0.004 + 0.004 * np.abs(want) + 2.0 ** -8 * np.abs(want)), what
    assert_rms_close(got, want, what)


@pytest.mark.parametrize("partitions", [1, 3])
def test_packed_attention_short_contexts_reversed_table(cuda, ops, partitions):
    """crates/qwc-cuda/tests/paged_attention.rs:10-131: contexts 23 and 257, page 64, reversed table."""
    case = synth.attention_case(11, [23, 257], page_size=64)
    for b in range(2):
        n = int((case["contexts"][b] + 63) // 64)
        case["block_tables"][b, :n] = case["block_tables"][b, :n][::-1].copy()
    check_attention(run_attention(cuda, ops, case, 64, partitions), attention_oracle(case, 64), "ctx 23/257")


@pytest.mark.parametrize("page_size,partitions", [(64, 1), (64, 5), (16, 1), (16, 8)],
                         ids=["page64_reference_shape", "page64_split_reference_shape",
                              "page16_oracle_generalisation", "page16_split_oracle_generalisation"])
def test_packed_attention_ragged_rows(cuda, ops, page_size, partitions):
    """crates/qwc-cuda/tests/paged_attention.rs:950-973: ragged rows with per-row permuted tables."""
    case = synth.attention_case(12, [1, 63, 64, 65, 3000, 777, 4096], page_size=page_size, with_gate=True)
    check_attention(run_attention(cuda, ops, case, page_size, partitions), attention_oracle(case, page_size),
                    f"ragged page {page_size} P{partitions}")


def test_packed_attention_benchmark_config_page16_scaled_oracle_generalisation_no_reference_test(cuda, ops):
    """Benchmark config 1: 32 sequences, contexts uniform in [128, 2048], page 16, per-head KV scale."""
    contexts = synth.uniform_contexts(0, 32, 128, 2048)
    case = synth.attention_case(0, contexts, page_size=16, with_gate=False, scaled=True)
    want = attention_oracle(case, 16)
    for partitions in (1, 4):
        check_attention(run_attention(cuda, ops, case, 16, partitions), want, f"config 1 P{partitions}")


def test_packed_attention_split_matches_unsplit_and_oversized_workspace(cuda, ops):
    """crates/qwc-cuda/tests/paged_attention.rs:977-1031 and :735-764."""
    torch = cuda
    case = synth.attention_case(13, [2048, 300, 5000], page_size=16, with_gate=True)
    unsplit = run_attention(torch, ops, case, 16, 1)
    split = run_attention(torch, ops, case, 16, 7)
    assert np.max(np.abs(unsplit - split)) <= 0.004 + 0.01 * np.max(np.abs(unsplit))
    # more partitions than 16-token units for the short row: empty partitions must merge cleanly
    many = run_attention(torch, ops, case, 16, 40)
    assert np.max(np.abs(unsplit - many)) <= 0.004 + 0.01 * np.max(np.abs(unsplit))


def test_packed_attention_sharp_softmax(cuda, ops):
    """crates/qwc-cuda/tests/paged_attention.rs:1038-1099: one key dominates the softmax."""
    case = synth.attention_case(14, [900], page_size=16)
    keys = synth.e4m3_decode(case["key_cache"])
    page = case["block_tables"][0, 411 // 16]
    query = synth.bf16_value(case["query"])
    for kv in range(4):
        boost = np.mean(query[0, kv * 6:(kv + 1) * 6], axis=0)
        keys[page, kv, 411 % 16] = np.clip(boost * 40.0, -448, 448)
    case["key_cache"] = synth.e4m3_encode(keys)
    got = run_attention(cuda, ops, case, 16, 2)
    want = attention_oracle(case, 16)
    scale = np.max(np.abs(want))
    assert np.max(np.abs(got - want)) <= 0.006 * scale + 0.004


@pytest.mark.parametrize("contexts,page_size,partitions", [
    ([16, 1, 0, 127, 128, 129], 16, 2),          # stages of one unit, of a whole stage and of one unit more
    ([30000, 33, 0, 31001, 17, 30016, 29999], 16, 40),   # 200 units per SM: large chunks and two small ones each
    ([60000, 1, 70001, 64, 65000, 60064, 60001], 64, 200),  # 530 units: three small ones
    ([60000, 70001, 500], 16, 2),                # the workspace has two slots per row: no chunk below a row's length
], ids=["short", "two_small", "three_small", "two_slots"])
def test_packed_attention_chunks(cuda, ops, contexts, page_size, partitions):
    """Every cut of the line into chunks, with rows without context; the slots that no piece is written to hold NaN
    before the call (rows share their pages: what is tested is the plan)."""
    torch = cuda
    case = synth.attention_case(16, [1024], page_size=page_size)
    contexts = np.asarray(contexts, dtype=np.uint32)
    blocks = (int(contexts.max()) + page_size - 1) // page_size + 1
    rng = np.random.default_rng(16)
    case.update(contexts=contexts, max_blocks=blocks, batch=contexts.size,
                block_tables=rng.integers(0, case["num_blocks"], (contexts.size, blocks)).astype(np.uint32),
                query=synth.bf16_bits(rng.standard_normal((contexts.size, 24, 256), dtype=np.float32)))
    out = bf16_out(torch, contexts.size, 24, 256)
    workspace = torch.full((ops.packed_workspace_bytes(contexts.size, partitions),), 0xFF, dtype=torch.uint8, device="cuda")
    ops.gated_packed(dev(torch, case["query"]), None, dev(torch, case["key_cache"]), dev(torch, case["value_cache"]),
                     dev(torch, case["block_tables"]), dev(torch, contexts), blocks, out, contexts.size, 0, partitions,
                     workspace, page_size, None, None)
    torch.cuda.synchronize()
    got, want = synth.bf16_value(host(out)), attention_oracle(case, page_size)
    want[contexts == 0] = 0.0  # (the oracle divides by a sum of nothing)
    check_attention(got, want, "chunks")


@pytest.mark.parametrize("contexts,table_tokens", [([2048, 300, 1, 0, 777, 128, 129, 1500, 90], 32768),
                                                   ([30000, 33, 0, 31001, 17, 30016, 29999], 32768)],
                         ids=["no_small_chunk_has_work", "two_small"])
def test_packed_attention_chunks_claimed_beside_another_stream(cuda, ops, contexts, table_tokens):
    """Chunks are claimed while calls on another stream hold SMs: whoever is first takes them, and the outputs, gated
    and scaled, are the same bits as alone (what a piece is does not depend on who works on it)."""
    torch = cuda
    contexts = np.asarray(contexts, dtype=np.uint32)
    rows, blocks, partitions = contexts.size, table_tokens // 16, 128
    case = synth.attention_case(21, [1024], page_size=16, scaled=True)
    rng = np.random.default_rng(21)
    tables = rng.integers(0, case["num_blocks"], (rows, blocks)).astype(np.uint32)
    query = synth.bf16_bits(rng.standard_normal((rows, 24, 256), dtype=np.float32))
    gate = synth.bf16_bits(rng.standard_normal((rows, 24, 512), dtype=np.float32))
    keys, values, tables_d, query_d, gate_d, contexts_d, ks, vs = (
        dev(torch, a) for a in (case["key_cache"], case["value_cache"], tables, query, gate, contexts, case["k_scale"],
                                case["v_scale"]))
    full_d = dev(torch, np.full(rows, table_tokens, dtype=np.uint32))
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    workspaces = [torch.full((ops.packed_workspace_bytes(rows, partitions),), 0xFF, dtype=torch.uint8, device="cuda")
                  for _ in streams]
    outs = [bf16_out(torch, rows, 24, 256) for _ in range(9)]
    busy = bf16_out(torch, rows, 24, 256)

    def call(lengths, out, workspace):
        ops.gated_packed(query_d, gate_d, keys, values, tables_d, lengths, blocks, out, rows, 0, partitions, workspace, 16,
                         ks, vs)

    torch.cuda.synchronize()
    call(contexts_d, outs[0], workspaces[0])
    torch.cuda.synchronize()
    for out in outs[1:]:
        with torch.cuda.stream(streams[1]):
            call(full_d, busy, workspaces[1])
        with torch.cuda.stream(streams[0]):
            call(contexts_d, out, workspaces[0])
    torch.cuda.synchronize()
    for out in outs[1:]:
        assert torch.equal(out, outs[0])
    want = attention_oracle(dict(case, contexts=contexts, block_tables=tables, max_blocks=blocks, query=query,
                                 gate_projection=gate), 16)
    want[contexts == 0] = 0.0  # (the oracle divides by a sum of nothing)
    check_attention(synth.bf16_value(host(outs[0])), want, "two streams")


def test_packed_attention_positions_beyond_32_bits(cuda, ops):
    """A block table that could describe 134 million tokens, with two slots per row: the plan's positions no longer
    fit 32 bits."""
    torch = cuda
    case = synth.attention_case(17, [700, 3], page_size=64)
    blocks = 1 << 21
    tables = torch.zeros((2, blocks), dtype=torch.int32, device="cuda")
    tables[:, :case["max_blocks"]] = dev(torch, case["block_tables"].astype(np.int32))
    out = bf16_out(torch, 2, 24, 256)
    workspace = torch.zeros(ops.packed_workspace_bytes(2, 2), dtype=torch.uint8, device="cuda")
    ops.gated_packed(dev(torch, case["query"]), None, dev(torch, case["key_cache"]), dev(torch, case["value_cache"]),
                     tables, dev(torch, case["contexts"]), blocks, out, 2, 0, 2, workspace, 64, None, None)
    torch.cuda.synchronize()
    check_attention(synth.bf16_value(host(out)), attention_oracle(case, 64), "wide plan")


@pytest.mark.parametrize("kind", ["tiny", "large", "outlier", "spread"])
def test_packed_attention_query_digits(cuda, ops, kind):
    """Queries far from unit scale.  The e4m3 digits of a query hold a bf16 exactly down to 2^-32 of the binade of its
    head's largest element, so the bounds are those of every attention test."""
    case = synth.attention_case(18, [300, 41], page_size=16, with_gate=True)
    query = synth.bf16_value(case["query"]).astype(np.float32)
    rng = np.random.default_rng(18)
    if kind == "tiny":
        query *= np.float32(2.0 ** -12)
    elif kind == "large":  # the scores stay moderate: four dims of each head
        query *= (rng.random(query.shape) < 4 / 256) * np.float32(8.0)
    elif kind == "outlier":  # one dim 4096 times the others, on keys that are zero there
        query[:, :, 7] = 4096.0
        keys = synth.e4m3_decode(case["key_cache"])
        keys[..., 7] = 0.0
        case["key_cache"] = synth.e4m3_encode(keys)
    else:
        query *= np.exp2(-rng.integers(0, 24, query.shape)).astype(np.float32)
    case["query"] = synth.bf16_bits(query)
    for partitions in (1, 3):
        check_attention(run_attention(cuda, ops, case, 16, partitions), attention_oracle(case, 16), kind)


@pytest.mark.parametrize("long_tokens,rows,partitions", [(6 << 20, 75, 1), (400 << 20, 1, 1000)],
                         ids=["three_whole_pairs_on_one_sm", "small_chunks"])
def test_packed_attention_waits_longer_than_their_limit_while_the_stream_goes_on(cuda, ops, long_tokens, rows,
                                                                                 partitions):
    """Contexts of millions of tokens, on which the query of the task after the next and the next list of tasks are
    waited for longer than the 20 ms in which a wait gives up when nothing moves.  All of a row's table names one page,
    so that the result is attention over that page."""
    torch = cuda
    case = synth.attention_case(22, [64] * rows, page_size=64, with_gate=True)
    blocks = long_tokens // 64
    contexts = np.full(rows, 64, dtype=np.uint32)
    contexts[0::37] = long_tokens  # (pairs are dealt round the SMs: with 148 of them these rows meet on four)
    tables = dev(torch, case["block_tables"][:, :1].astype(np.int32)).repeat(1, blocks)
    out = bf16_out(torch, rows, 24, 256)
    workspace = torch.zeros(max(16, ops.packed_workspace_bytes(rows, partitions)), dtype=torch.uint8, device="cuda")
    ops.gated_packed(dev(torch, case["query"]), dev(torch, case["gate_projection"]), dev(torch, case["key_cache"]),
                     dev(torch, case["value_cache"]), tables, dev(torch, contexts), blocks, out, rows, 0, partitions,
                     workspace, 64, None, None)
    torch.cuda.synchronize()
    assert ops.abi.lib.qwc_device_status() == 0
    check_attention(synth.bf16_value(host(out)), attention_oracle(case, 64), "long waits")


@pytest.mark.parametrize("binades", [0, 13, 14, 18, 20, 22, 25, 28, 31, 32])
def test_packed_attention_query_holds_what_f16_holds(cuda, ops, binades):
    """One dim of 2^15, on keys that are zero there, beside dims that decide the softmax, from the same binade down to
    2^-17: f16 holds all of these exactly (eight significant bits), and so must the digits of the query.  The bounds are
    those of every attention test; a query of three digits 2^-4 apart misses them from 2^18 on."""
    case = synth.attention_case(20, [300, 41], page_size=16, scaled=True)
    rng = np.random.default_rng(binades)
    small = 2.0 ** (15 - binades)
    codes = rng.integers(128, 256, (2, 24, 256)) * rng.choice([-1.0, 1.0], (2, 24, 256))  # eight significant bits each
    query = (codes / 128.0 * small).astype(np.float32)
    query[:, :, 7] = 2.0 ** 15
    keys = rng.standard_normal(case["key_cache"].shape, dtype=np.float32)
    keys[..., 7] = 0.0
    # scores of order 1: 256 products of about 1.5 small, over 16
    case.update(query=synth.bf16_bits(query), key_cache=synth.e4m3_encode(keys),
                k_scale=np.full(4, 1.0 / small, dtype=np.float32))
    for partitions in (1, 3):
        check_attention(run_attention(cuda, ops, case, 16, partitions), attention_oracle(case, 16), f"2^{binades}")


@pytest.mark.parametrize("value", [np.nan, np.inf])
def test_packed_attention_non_finite_query_stays_in_its_head(cuda, ops, value):
    case = synth.attention_case(19, [300, 41], page_size=16)
    clean = run_attention(cuda, ops, case, 16, 3)
    query = synth.bf16_value(case["query"]).astype(np.float32)
    query[0, 8, 100] = value
    got = run_attention(cuda, ops, dict(case, query=synth.bf16_bits(query)), 16, 3)
    same = np.ones((2, 24), dtype=bool)
    same[0, 8] = False
    assert np.array_equal(got[same], clean[same])
    assert not np.array_equal(got[0, 8], clean[0, 8])


@pytest.mark.parametrize("contexts,partitions,share", [(range(29, 73), 1, 0.02), (range(128, 2048, 60), 16, 0.09)],
                         ids=["undivided", "split"])
def test_packed_attention_is_nearly_the_rounded_exact_result(cuda, ops, contexts, partitions, share):
    """How many outputs are not the float64 result rounded to bf16.  Measured 0.9 % undivided (a probability is kept to
    2^-13, so an element is off by that over the square root of its tokens, and crosses a rounding boundary every
    hundredth time) and 7.2 % split (the partials are f16); the f16 operands that the digits have taken the place of
    gave 8.2 % and 11.5 %."""
    case = synth.attention_case(24, list(contexts), page_size=16, scaled=True)
    keys, values = synth.e4m3_decode(case["key_cache"]).astype(np.float64), synth.e4m3_decode(case["value_cache"])
    query = synth.bf16_value(case["query"]).astype(np.float64)
    want = np.zeros(query.shape)
    for row, context in enumerate(case["contexts"].astype(int)):
        pages = case["block_tables"][row, :(context + 15) // 16]
        for kv in range(4):
            k, v = (cache[pages, kv].reshape(-1, 256)[:context] * np.float64(scale[kv])
                    for cache, scale in ((keys, case["k_scale"]), (values, case["v_scale"])))
            scores = query[row, 6 * kv:6 * kv + 6] @ k.T / 16.0
            weights = np.exp(scores - scores.max(axis=1, keepdims=True))
            want[row, 6 * kv:6 * kv + 6] = weights / weights.sum(axis=1, keepdims=True) @ v
    got = run_attention(cuda, ops, case, 16, partitions)
    assert np.mean(got != cuda.from_numpy(want).to(cuda.bfloat16).float().numpy()) < share


@pytest.mark.parametrize("partitions", [1, 3])
def test_packed_attention_staged_output_holds_the_bf16_output(cuda, ops, partitions):
    """The staged f16 output is the bf16 output, NaN for NaN (of a gate, and of a query whose scores are infinite);
    values beyond f16 saturate."""
    from qwencore_b200 import abi

    torch = cuda
    case = synth.attention_case(23, [300, 41], page_size=16, with_gate=True, scaled=True)
    query = synth.bf16_value(case["query"]).astype(np.float32)
    query[0, 8, 100] = np.inf
    gate = synth.bf16_value(case["gate_projection"]).astype(np.float32)
    gate[1, 3, 256 + 7] = np.nan
    v_scale = case["v_scale"].copy()
    v_scale[3] *= 1e7  # the heads of the last kv head reach beyond 65504
    out, staged = bf16_out(torch, 2, 24, 256), ops.new_staged(2, 24 * 256)
    workspace = torch.zeros(max(16, ops.packed_workspace_bytes(2, partitions)), dtype=torch.uint8, device="cuda")
    held = [dev(torch, a) for a in (synth.bf16_bits(query), synth.bf16_bits(gate), case["key_cache"],
                                    case["value_cache"], case["block_tables"], case["contexts"], case["k_scale"], v_scale)]
    abi.check(abi.lib.qwc_paged_attention_packed_fp8_staged(
        *[a.data_ptr() for a in held], out.data_ptr(), staged.data_ptr(), workspace.data_ptr(), workspace.numel(), 2, 0,
        case["max_blocks"], 16, 0, partitions, 1.0 / 16.0, torch.cuda.current_stream().cuda_stream), "staged")
    torch.cuda.synchronize()
    want = synth.bf16_value(host(out)).reshape(2, 24 * 256)
    got = host(ops.unstage(staged, 2, 24 * 256)).astype(np.float32)
    assert np.isnan(want[0, 8 * 256:9 * 256]).all() and np.isnan(want[1, 3 * 256 + 7])
    assert np.count_nonzero(np.abs(want) > 65504) > 100  # (infinities where f16 partials have been merged)
    assert np.array_equal(got, np.clip(want, -65504, 65504).astype(np.float16).astype(np.float32), equal_nan=True)


@pytest.mark.parametrize("partitions", [1, 4])
def test_packed_attention_non_finite_value_stays_in_its_row(cuda, ops, partitions):
    """Rows whose stages are partly filled, on CTAs that have had full stages of a row with NaN values before."""
    contexts = np.full(150, 16, dtype=np.uint32)
    contexts[:37] = 1024  # (with 148 SMs undivided rows 37 apart meet on a CTA)
    case = synth.attention_case(25, contexts, page_size=16)
    clean = run_attention(cuda, ops, case, 16, partitions)
    values = case["value_cache"].copy()
    values[case["block_tables"][0, :64]] = 0x7F
    got = run_attention(cuda, ops, dict(case, value_cache=values), 16, partitions)
    assert np.isnan(got[0]).all()
    assert np.array_equal(got[1:], clean[1:])


def test_packed_attention_legacy_entry_uses_configured_page_size(cuda, ops):
    from qwencore_b200 import abi

    torch = cuda
    case = synth.attention_case(15, [70, 129], page_size=64, with_gate=True)
    before = abi.get_shape()
    try:
        abi.configure(before[0], 64)
        out = bf16_out(torch, 2, 24, 256)
        ops.gated_packed_legacy(dev(torch, case["query"]), dev(torch, case["gate_projection"]),
                                dev(torch, case["key_cache"]), dev(torch, case["value_cache"]),
                                dev(torch, case["block_tables"]), dev(torch, case["contexts"]), case["max_blocks"],
                                out, 2, 0, 1, None)
        torch.cuda.synchronize()
        check_attention(synth.bf16_value(host(out)), attention_oracle(case, 64), "legacy entry")
        with pytest.raises(abi.QwcError) as error:  # segment tiles are prefill shapes
            ops.gated_packed_legacy(dev(torch, case["query"]), None, dev(torch, case["key_cache"]),
                                    dev(torch, case["value_cache"]), dev(torch, case["block_tables"]),
                                    dev(torch, case["contexts"]), case["max_blocks"], out, 2, 0, 1, None, tile_size=32)
        assert error.value.code == abi.CUDA_ERROR_NOT_SUPPORTED
        with pytest.raises(abi.QwcError) as error:  # workspace too small (paged_attention.cu:1876-1880)
            ops.gated_packed_legacy(dev(torch, case["query"]), None, dev(torch, case["key_cache"]),
                                    dev(torch, case["value_cache"]), dev(torch, case["block_tables"]),
                                    dev(torch, case["contexts"]), case["max_blocks"], out, 2, 0, 4,
                                    torch.zeros(16, dtype=torch.uint8, device="cuda"))
        assert error.value.code == abi.CUDA_ERROR_INVALID_VALUE
    finally:
        abi.configure(*before)


# ---------------------------------------------------------------------------------------
# Gated DeltaNet int8 step
# ---------------------------------------------------------------------------------------

def run_delta(torch, ops, case, batch, v_heads, beta=None):
    from qwencore_b200 import abi

    before = abi.get_shape()
    abi.configure(v_heads, before[1])
    try:
        state = dev(torch, case["state"])
        scales = dev(torch, case["scales"])
        out = torch.zeros((batch, v_heads, 128), dtype=torch.float32, device="cuda")
        ops.delta_decode_slots_packed(state, scales, dev(torch, case["slots"]), dev(torch, case["q"]),
                                      dev(torch, case["k"]), dev(torch, case["v"]), dev(torch, case["alpha"]),
                                      dev(torch, case["beta"] if beta is None else beta), dev(torch, case["kq"]), out,
                                      case["capacity"], batch)
        torch.cuda.synchronize()
        return host(state), host(scales), host(out)
    finally:
        abi.configure(*before)


@pytest.mark.parametrize("batch,v_heads", [(32, 32), (1, 32), (5, 48)],
                         ids=["b32_h32_oracle_generalisation", "b1_h32_oracle_generalisation", "b5_h48_reference_shape"])
def test_delta_decode_int8_matches_oracle(cuda, ops, batch, v_heads):
    """Benchmark config 2 (32 slots, 32 value heads) and the reference's 48-head shape."""
    case = synth.delta_case(2, batch, v_heads)
    want_state, want_scales = case["state"].copy(), case["scales"].copy()
    want_out = oracle.delta_decode_int8(want_state, want_scales, case["slots"], case["q"], case["k"], case["v"],
                                        case["alpha"], case["beta"], case["kq"], batch, v_heads)
    state, scales, out = run_delta(cuda, ops, case, batch, v_heads)
    # out is read as bf16 downstream (cuda/delta_output.cu:38)
    assert_rms_close(oracle.bf16_round(out), oracle.bf16_round(want_out), "delta out")
    # reference: output within 2e-3 relative (crates/qwc-cuda/tests/delta_net.rs:113-135)
    assert np.max(np.abs(out - want_out)) <= 2e-3 * np.max(np.abs(want_out))
    # state: the fp32 summation order of u differs, so a code may move by one step on a few elements
    diff = np.abs(state.astype(np.int32) - want_state.astype(np.int32))
    assert diff.max() <= 1
    assert np.mean(diff > 0) < 0.02
    assert np.allclose(scales, want_scales, rtol=1e-5, atol=0)
    untouched = sorted(set(range(case["capacity"])) - set(case["slots"].tolist()))
    for slot in untouched:  # crates/qwc-cuda/tests/delta_net.rs:184-245
        assert np.array_equal(state[slot], case["state"][slot])
        assert np.array_equal(scales[slot], case["scales"][slot])


@pytest.mark.parametrize("batch,v_heads", [("last_four_lanes", 32), ("first_eight_lanes", 32), ("last_four_lanes", 48),
                                           ("first_eight_lanes", 48), (32, 32), (32, 48), (1, 32), (2, 32), (3, 48)],
                         ids=["last_four_lanes", "first_eight_lanes", "last_four_lanes_h48", "first_eight_lanes_h48",
                              "full_batch", "full_batch_h48", "row_split_16", "row_split_8", "row_split_4"])
@pytest.mark.parametrize("exponent", [0, -100, 92], ids=["unit_q", "tiny_q", "huge_q"])
def test_delta_decode_both_forms(cuda, ops, batch, v_heads, exponent):
    """On either side of the line between four and eight lanes per row (five CTAs per SM; with 148 SMs 23 | 24 rows of
    32 heads and 15 | 16 of 48), at the full batch, with row splits, with a key of zeros
    and with a query at the ends of the fp32 range (a power of two: only `out` scales with it, the update
    does not see q).  Bounds: out within 1e-5 of its row's largest value (128 fp32 roundings of 6e-8 on either
    side, in different orders), codes within one step, where row . k moves by a unit in the last place."""
    line = 5 * cuda.cuda.get_device_properties(0).multi_processor_count // v_heads
    if isinstance(batch, str):
        batch = line if batch == "last_four_lanes" else line + 1
        assert 3 < batch <= 32, "both forms have a batch of their own"
    case = synth.delta_case(11, batch, v_heads)
    k, q = case["k"].copy(), case["q"].copy()
    k[0] = 0.0
    q[batch - 1] = np.ldexp(q[batch - 1], exponent)
    case = dict(case, k=k, q=q, kq=np.einsum("bhd,bhd->bh", q, k).astype(np.float32))
    want_state, want_scales = case["state"].copy(), case["scales"].copy()
    want_out = oracle.delta_decode_int8(want_state, want_scales, case["slots"], case["q"], case["k"], case["v"],
                                        case["alpha"], case["beta"], case["kq"], batch, v_heads)
    state, scales, out = run_delta(cuda, ops, case, batch, v_heads)
    row_peak = np.max(np.abs(want_out), axis=(1, 2), keepdims=True)
    assert np.all(np.abs(out - want_out) <= 1e-5 * row_peak)
    diff = np.abs(state.astype(np.int32) - want_state.astype(np.int32))
    assert diff.max() <= 1 and np.mean(diff > 0) < 1e-4
    assert np.allclose(scales, want_scales, rtol=1e-5, atol=0)


@pytest.mark.parametrize("batch,v_heads", [(1, 48), (23, 32), (24, 32)],
                         ids=["row_split", "last_four_lanes", "first_eight_lanes"])
@pytest.mark.parametrize("before", [0, 0xFFFFFFFF], ids=["another_slot", "no_slot"])
def test_delta_slots_and_state_written_just_before_the_call(cuda, ops, batch, v_heads, before):
    """The kernel looks at a row's slot before the work ahead of it on the stream has ended, to have the tile
    brought into L2; what counts is what stands there afterwards.  Slots, state and scales are written by copies
    right before the call: the same bits as with everything in place long before."""
    torch = cuda
    from qwencore_b200 import abi

    case = synth.delta_case(13, batch, v_heads)
    want = run_delta(torch, ops, case, batch, v_heads)
    shape = abi.get_shape()
    abi.configure(v_heads, shape[1])
    try:
        fresh = [dev(torch, case[name]) for name in ("state", "scales", "slots")]
        vectors = [dev(torch, case[name]) for name in ("q", "k", "v", "alpha", "beta", "kq")]
        state, scales = torch.zeros_like(fresh[0]), torch.zeros_like(fresh[1])
        slots = dev(torch, np.full(batch, before, dtype=np.uint32))
        out = torch.zeros((batch, v_heads, 128), dtype=torch.float32, device="cuda")
        torch.cuda.synchronize()
        for target, source in zip((state, scales, slots), fresh):
            target.copy_(source)
        ops.delta_decode_slots_packed(state, scales, slots, *vectors, out, case["capacity"], batch)
        torch.cuda.synchronize()
    finally:
        abi.configure(*shape)
    for got, expected in zip((state, scales, out), want):
        assert np.array_equal(host(got), expected)
    assert abi.lib.qwc_device_status() == 0


@pytest.mark.parametrize("batch,v_heads", [(3, 32), (24, 32)], ids=["four_lanes", "eight_lanes"])
@pytest.mark.parametrize("vector", ["k", "q"])
def test_delta_dot_products_keep_small_elements_beside_an_outlier(cuda, ops, batch, v_heads, vector):
    """k (then q) holds a 1 where every state row's code is 0, and elements of 1e-5 to 1e-8 elsewhere: the dot
    product is the sum of the small ones alone.  The other inputs are chosen so that `out` is that dot product
    times a gate: v = 0 and q the unit vector of the outlier's column (out = -alpha beta row . k), or k = 0
    (out = alpha row . q).  Bound against float64: one rounding of each state element and at most 24 of the
    sum (16 in a lane, its two halves, three exchanges, the gates), 2^-24 of the sum of magnitudes each."""
    case = synth.delta_case(13, batch, v_heads)
    rng = synth.generator(13, "outlier")
    column = 77
    state = case["state"].copy()
    state[..., column] = 0
    x = (rng.choice([-1.0, 1.0], (batch, 16, 128)) * 10.0 ** rng.uniform(-8, -5, (batch, 16, 128))).astype(np.float32)
    x[..., column] = 1.0
    unit, zero = np.zeros_like(x), np.zeros_like(x)
    unit[..., column] = 1.0
    k, q = (x, unit) if vector == "k" else (zero, x)
    kq = np.full((batch, 16), 1.0 if vector == "k" else 0.0, dtype=np.float32)
    case = dict(case, state=state, k=k, q=q, kq=kq, v=np.zeros_like(case["v"]))
    _, _, out = run_delta(cuda, ops, case, batch, v_heads)
    rows = state[case["slots"]].astype(np.float64) * case["scales"][case["slots"]].astype(np.float64)[..., None]
    terms = rows * np.repeat(x.astype(np.float64), v_heads // 16, axis=1)[:, :, None, :]
    gate = case["alpha"].astype(np.float64) * (-case["beta"].astype(np.float64) if vector == "k" else 1.0)
    want = gate[..., None] * terms.sum(-1)
    bound = 25 * 2.0 ** -24 * np.abs(gate)[..., None] * np.abs(terms).sum(-1)
    assert np.all(np.abs(out - want) <= bound)


@pytest.mark.parametrize("batch", [3, 24], ids=["four_lanes", "eight_lanes"])
@pytest.mark.parametrize("value", [np.nan, np.inf])
def test_delta_non_finite_key_stays_in_its_head(cuda, ops, value, batch):
    v_heads = 32
    case = synth.delta_case(12, batch, v_heads)
    k = case["k"].copy()
    k[1, 4, 17] = value
    _, _, clean = run_delta(cuda, ops, case, batch, v_heads)
    _, _, out = run_delta(cuda, ops, dict(case, k=k), batch, v_heads)
    hit = np.zeros((batch, v_heads), dtype=bool)
    hit[1, 8:10] = True  # two value heads per key head
    assert not np.isfinite(out[hit]).any()
    assert np.array_equal(out[~hit], clean[~hit])


def test_delta_requantiser_is_bit_exact(cuda, ops):
    """beta = 0 makes every fp32 row value alpha * s exactly (tests/delta_net.rs:138-182), so the
    int8 codes and scales must equal the oracle's bit for bit."""
    batch, v_heads = 7, 32
    case = synth.delta_case(4, batch, v_heads, capacity=9)
    beta = np.zeros_like(case["beta"])
    want_state, want_scales = case["state"].copy(), case["scales"].copy()
    want_out = oracle.delta_decode_int8(want_state, want_scales, case["slots"], case["q"], case["k"], case["v"],
                                        case["alpha"], beta, case["kq"], batch, v_heads)
    state, scales, out = run_delta(cuda, ops, case, batch, v_heads, beta=beta)
    assert np.array_equal(state, want_state)
    assert np.array_equal(scales.view(np.uint32), want_scales.view(np.uint32))
    assert np.allclose(out, want_out, rtol=1e-4, atol=1e-6)


def test_delta_zero_rows_store_zero_scale(cuda, ops):
    batch, v_heads = 2, 32
    case = synth.delta_case(5, batch, v_heads, capacity=2)
    case["state"][:] = 0
    case["scales"][:] = 0
    case["v"][:] = 0
    state, scales, out = run_delta(cuda, ops, case, batch, v_heads)
    assert not state.any() and not scales.any() and not out.any()


def test_delta_slot_beyond_the_pool_is_skipped_and_reported(cuda, ops):
    """A row that names a state slot past the pool touches no memory: the kernel skips the row and
    the sticky status word tells the host (nothing faults; the access never happens)."""
    from qwencore_b200 import abi

    batch, v_heads = 3, 32
    case = synth.delta_case(6, batch, v_heads, capacity=4)
    slots = case["slots"].copy()
    bad_row = 1
    slots[bad_row] = 4  # capacity is 4: slots 0..3 exist
    case = dict(case, slots=slots)
    assert abi.lib.qwc_device_status() == 0
    try:
        state, scales, out = run_delta(cuda, ops, case, batch, v_heads)
        assert abi.lib.qwc_device_status() == 0x105
        # the pool is as it was wherever the rows in range did not write, and the bad row wrote nothing
        touched = {int(s) for i, s in enumerate(slots) if i != bad_row}
        for slot in range(case["capacity"]):
            if slot not in touched:
                assert np.array_equal(state[slot], case["state"][slot])
        assert not out[bad_row].any()
    finally:
        assert abi.lib.qwc_device_status_reset() == 0
    assert abi.lib.qwc_device_status() == 0


# ---------------------------------------------------------------------------------------
# Step glue
# ---------------------------------------------------------------------------------------

def test_rmsnorm_bf16_with_and_without_residual(cuda, ops):
    torch = cuda
    batch, hidden = 5, 5120
    x = synth.normal_bf16(6, "x", (batch, hidden))
    res = synth.normal_bf16(6, "res", (batch, hidden), std=3.0)
    w = synth.normal_bf16(6, "w", (hidden,), std=0.02)
    for with_residual in (False, True):
        res_want = res.copy()
        want = oracle.rmsnorm_bf16(x, res_want if with_residual else None, w, batch, hidden)
        res_dev = dev(torch, res)
        out = bf16_out(torch, batch, hidden)
        ops.rmsnorm_bf16(dev(torch, x), res_dev if with_residual else None, dev(torch, w), out, batch, hidden)
        torch.cuda.synchronize()
        if with_residual:  # the residual sum is one bf16 rounding: bit-exact
            assert np.array_equal(host(res_dev), res_want)
        got = synth.bf16_value(host(out))
        want_values = synth.bf16_value(want)
        assert np.max(np.abs(got - want_values)) <= 2.0 ** -7 * np.max(np.abs(want_values))
        assert_rms_close(got, want_values, "rmsnorm")


def test_fp8_embedding_gather_is_bit_exact(cuda, ops):
    torch = cuda
    vocab, cols = 1000, 512
    rows = synth.normal_bf16(7, "emb", (vocab, cols), std=0.02)
    table, scales = oracle.fp8_quantize_rows(rows, vocab, cols)
    tokens = np.array([0, 999, 17, 1000, 4000000000], dtype=np.uint32)  # last two are out of vocabulary
    want = oracle.fp8_embedding_gather(table, scales, tokens, cols, vocab)
    out = bf16_out(torch, tokens.size, cols)
    ops.fp8_embedding_gather(dev(torch, table), dev(torch, scales), dev(torch, tokens), out, tokens.size, cols, vocab)
    torch.cuda.synchronize()
    assert np.array_equal(host(out), want)
    assert not host(out)[3:].any()


# 5003: not a multiple of the row tile nor of the 16-byte store (the mma.sync kernel at every batch size);
# 5000: stores aligned, a ragged last tile (above eight rows the tcgen05 kernel); 12000: a table large
# enough that the tcgen05 kernel takes every batch size.
@pytest.mark.parametrize("batch,vocab", [(1, 5003), (8, 5003), (32, 5003), (8, 5000), (9, 5000), (16, 5000),
                                         (17, 5000), (32, 5000), (32, 4096), (1, 12000), (5, 12000)])
def test_fp8_lm_head_and_argmax(cuda, ops, batch, vocab):
    torch = cuda
    hidden = 5120
    rows = synth.normal_bf16(8, "head", (vocab, hidden), std=0.02)
    weights, scales = oracle.fp8_quantize_rows(rows, vocab, hidden)
    x = synth.normal_bf16(8, f"h{batch}", (batch, hidden))
    want = oracle.fp8_lm_head(weights, scales, x, batch, hidden, vocab)
    logits = torch.zeros((batch, vocab), dtype=torch.float32, device="cuda")
    ops.fp8_lm_head(dev(torch, weights), dev(torch, scales), dev(torch, x), logits, batch, hidden, vocab)
    parts = 64
    pv = torch.zeros(batch * parts, dtype=torch.float32, device="cuda")
    pi = u32_out(torch, batch * parts)
    tokens = u32_out(torch, batch)
    ops.argmax(logits, pv, pi, tokens, vocab, batch, parts)
    torch.cuda.synchronize()
    got = host(logits)
    assert_rms_close(got, want, "lm_head", bf16_grid=False)
    # argmax of the GPU logits is exact; against the oracle logits it agrees wherever the top-2 gap is clear
    assert np.array_equal(host(tokens), oracle.argmax(got, vocab, batch))
    ordered = np.sort(want, axis=1)
    clear = (ordered[:, -1] - ordered[:, -2]) > 4 * np.max(np.abs(got - want))
    assert np.array_equal(host(tokens)[clear], oracle.argmax(want, vocab, batch)[clear])


def test_argmax_ties_go_to_lower_index(cuda, ops):
    """crates/qwc-cuda/tests/sampling.rs:19-27"""
    torch = cuda
    vocab = 151936
    logits = np.full((7, vocab), -2.0, dtype=np.float32)
    logits[0, [150000, 77, 9000]] = 5.0
    logits[1, vocab - 1] = 1.0
    logits[2, :] = 0.25
    # what `value > best || (value == best && index < best_index)` does with the special values
    # (cuda/sampling.cu:11-14): a NaN never wins, -inf is an ordinary smallest value, -0 equals +0
    logits[3, :] = np.nan
    logits[4, :] = -np.inf
    logits[4, 5] = np.nan
    logits[5, :] = -np.inf
    logits[5, [70000, 120001]] = -3.0e38
    logits[6, :] = -1.0
    logits[6, 9] = 0.0
    logits[6, 4] = -0.0
    parts = 256
    pv = torch.zeros(7 * parts, dtype=torch.float32, device="cuda")
    pi = u32_out(torch, 7 * parts)
    tokens = u32_out(torch, 7)
    ops.argmax(dev(torch, logits), pv, pi, tokens, vocab, 7, parts)
    torch.cuda.synchronize()
    assert host(tokens).tolist() == [77, vocab - 1, 0, 0xFFFFFFFF, 0, 70000, 4]


@pytest.mark.parametrize("vocab", [1, 3, 37, 10240, 10243, 81921, 151938])
def test_argmax_any_width_and_alignment(cuda, ops, vocab):
    """Widths that fill a thread's batch of loads partly, wholly and more than once, rows on and off 16-byte
    boundaries, with many ties and NaNs."""
    torch = cuda
    rng = np.random.default_rng(vocab)
    logits = rng.integers(-3, 4, (5, vocab)).astype(np.float32)
    logits[rng.random((5, vocab)) < 0.2] = np.nan
    logits[3] = np.where(rng.random(vocab) < 0.5, -np.inf, np.nan)
    logits[4] = rng.permutation(vocab)
    want = []
    for row in logits:
        there = np.flatnonzero(~np.isnan(row))
        want.append(int(there[np.argmax(row[there])]) if there.size else 0xFFFFFFFF)
    tokens = u32_out(torch, 5)
    ops.argmax(dev(torch, logits), torch.zeros(5 * 256, dtype=torch.float32, device="cuda"), u32_out(torch, 5 * 256),
               tokens, vocab, 5, 256)
    torch.cuda.synchronize()
    assert host(tokens).tolist() == want


@pytest.mark.parametrize("vocab", [2 ** 31 - 1, 2 ** 31 - 4096])
def test_argmax_up_to_the_largest_width(cuda, ops, vocab):
    """The last columns that an int can count; nothing behind the row is read."""
    torch = cuda
    logits = torch.zeros(vocab, dtype=torch.float32, device="cuda")
    logits[vocab - 1] = 1.0
    tokens = u32_out(torch, 1)
    ops.argmax(logits, torch.zeros(256, dtype=torch.float32, device="cuda"), u32_out(torch, 256), tokens, vocab, 1, 256)
    torch.cuda.synchronize()
    assert host(tokens).tolist() == [vocab - 1]


@pytest.mark.parametrize("v_heads", [32, 48], ids=["h32_oracle_generalisation", "h48_reference_shape"])
def test_delta_prepare_and_gated_rmsnorm(cuda, ops, v_heads):
    """crates/qwc-cuda/tests/delta_net.rs:576-716 (CPU conv/gate check) and :716-777."""
    from qwencore_b200 import abi

    torch = cuda
    batch, capacity, k_heads, dim = 4, 6, 16, 128
    channels = 2 * k_heads * dim + v_heads * dim
    z_offset = channels
    a_offset = z_offset + v_heads * dim
    b_offset = a_offset + v_heads
    stride = b_offset + v_heads
    rng = synth.generator(9, f"prepare{v_heads}")
    mixed = synth.bf16_bits(rng.standard_normal((batch, stride), dtype=np.float32))
    conv_weight = synth.bf16_bits(rng.standard_normal((channels, 4), dtype=np.float32) * 0.5)
    a_log = synth.bf16_bits(rng.standard_normal(v_heads, dtype=np.float32) * 0.5)
    dt_bias = synth.bf16_bits(rng.standard_normal(v_heads, dtype=np.float32) * 0.5)
    conv_state = rng.standard_normal((capacity, channels, 3), dtype=np.float32)
    slots = rng.permutation(capacity)[:batch].astype(np.uint32)

    want_state = conv_state.copy()
    base = mixed.ctypes.data
    q, k, v, alpha, beta, kq = oracle.delta_prepare_decode(mixed, base + 2 * a_offset, base + 2 * b_offset, conv_weight,
                                                           a_log, dt_bias, want_state, slots, batch, stride, stride,
                                                           k_heads, v_heads)
    before = abi.get_shape()
    abi.configure(v_heads, before[1])
    try:
        d_mixed = dev(torch, mixed)
        d_state = dev(torch, conv_state)
        tq = torch.zeros((batch, k_heads, dim), dtype=torch.float32, device="cuda")
        tk = torch.zeros_like(tq)
        tv = torch.zeros((batch, v_heads, dim), dtype=torch.float32, device="cuda")
        ta = torch.zeros((batch, v_heads), dtype=torch.float32, device="cuda")
        tb = torch.zeros_like(ta)
        tkq = torch.zeros((batch, k_heads), dtype=torch.float32, device="cuda")
        ops.delta_prepare_decode(d_mixed, a_offset, b_offset, dev(torch, conv_weight), dev(torch, a_log),
                                 dev(torch, dt_bias), d_state, dev(torch, slots), tq, tk, tv, ta, tb, tkq, capacity,
                                 batch, stride)
        values = rng.standard_normal((batch, v_heads, dim), dtype=np.float32)
        weight = synth.bf16_bits(1.0 + 0.1 * rng.standard_normal(dim, dtype=np.float32))
        normed = bf16_out(torch, batch, v_heads, dim)
        ops.delta_gated_rmsnorm(dev(torch, values), d_mixed, z_offset, dev(torch, weight), normed, batch, stride)
        torch.cuda.synchronize()
    finally:
        abi.configure(*before)

    # history shift is a copy: bit-exact; untouched slots stay untouched
    assert np.array_equal(host(d_state), want_state)
    assert np.array_equal(host(tv), v)  # conv + SiLU snapped to bf16: allow no more than one bf16 step
    for got, want, name in [(tq, q, "q"), (tk, k, "k"), (ta, alpha, "alpha"), (tb, beta, "beta"), (tkq, kq, "kq")]:
        assert np.allclose(host(got), want, rtol=2e-3, atol=2e-6), name
    want_norm = oracle.delta_gated_rmsnorm(values, base + 2 * z_offset, weight, batch, v_heads, stride)
    got_norm = synth.bf16_value(host(normed))
    want_norm = synth.bf16_value(want_norm)
    assert np.max(np.abs(got_norm - want_norm)) <= 2.0 ** -6 * np.max(np.abs(want_norm))
    assert_rms_close(got_norm, want_norm, "gated rmsnorm", bound=2e-2)


@pytest.mark.parametrize("page_size,scaled", [(64, False), (16, True)],
                         ids=["page64_reference_shape", "page16_kv_scales_oracle_generalisation"])
def test_prepare_attention_writes_query_and_fp8_pages(cuda, ops, page_size, scaled):
    """crates/qwc-cuda/tests/attention_prepare.rs:9-33"""
    torch = cuda
    batch, num_blocks = 3, 7
    rng = synth.generator(10, f"attnprep{page_size}")
    query_gate = synth.bf16_bits(rng.standard_normal((batch, 24 * 512), dtype=np.float32))
    key_proj = synth.bf16_bits(rng.standard_normal((batch, 4 * 256), dtype=np.float32))
    value_proj = synth.bf16_bits(rng.standard_normal((batch, 4 * 256), dtype=np.float32))
    qw = synth.bf16_bits(rng.standard_normal(256, dtype=np.float32) * 0.1)
    kw = synth.bf16_bits(rng.standard_normal(256, dtype=np.float32) * 0.1)
    positions = np.array([0, 5 * page_size + 3, 2 * page_size + page_size - 1], dtype=np.uint32)
    cosine, sine = oracle.rope_rows(positions)
    physical = np.array([6, 2, 4], dtype=np.uint32)
    offsets = (positions % page_size).astype(np.uint32)
    k_scale = v_scale = None
    if scaled:
        k_scale = np.array([0.02, 0.03, 0.015, 0.025], dtype=np.float32)
        v_scale = np.array([0.01, 0.02, 0.03, 0.04], dtype=np.float32)
    key_cache = np.zeros((num_blocks, 4, page_size, 256), dtype=np.uint8)
    value_cache = np.zeros_like(key_cache)
    want_k, want_v = key_cache.copy(), value_cache.copy()
    want_q = oracle.prepare_attention_decode_fp8(query_gate, key_proj, value_proj, qw, kw, cosine, sine, physical,
                                                 offsets, want_k, want_v, batch, page_size, k_scale=k_scale,
                                                 v_scale=v_scale)
    d_k, d_v = dev(torch, key_cache), dev(torch, value_cache)
    query = bf16_out(torch, batch, 24, 256)
    ops.prepare_attention_decode(dev(torch, query_gate), dev(torch, key_proj), dev(torch, value_proj), dev(torch, qw),
                                 dev(torch, kw), dev(torch, cosine), dev(torch, sine), dev(torch, physical),
                                 dev(torch, offsets), query, d_k, d_v, batch, page_size, 24 * 512, 4 * 256, 4 * 256,
                                 None if k_scale is None else dev(torch, k_scale),
                                 None if v_scale is None else dev(torch, v_scale))
    torch.cuda.synchronize()
    got_q = synth.bf16_value(host(query))
    assert np.max(np.abs(got_q - synth.bf16_value(want_q))) <= 2.0 ** -6 * np.max(np.abs(got_q))
    got_k, got_v = host(d_k), host(d_v)
    # V is a pure bf16 -> e4m3 conversion: bit-exact without scales (with scales the reciprocal may differ by an ulp)
    if not scaled:
        assert np.array_equal(got_v, want_v)
    for got, want in ((got_k, want_k), (got_v, want_v)):
        written = want != 0
        assert np.array_equal(got != 0, written) or np.mean((got != 0) != written) < 1e-3
        steps = np.abs(got.astype(np.int32) - want.astype(np.int32))
        assert steps.max() <= 1 and np.mean(steps > 0) < 0.02  # rsqrt vs 1/sqrt may move a code by one


# ---------------------------------------------------------------------------------------
# Device-side batch packing (bit-exact)
# ---------------------------------------------------------------------------------------

def packing_case(seed, capacity, max_blocks, page_size, live):
    rng = synth.generator(seed, "packing")
    seq_tokens = np.zeros(capacity, dtype=np.uint32)
    seq_blocks = np.zeros((capacity, max_blocks), dtype=np.uint32)
    counts = np.zeros(capacity, dtype=np.uint32)
    pool = rng.permutation(capacity * max_blocks).astype(np.uint32)
    cursor = 0
    slots = rng.permutation(capacity)[:live]
    for slot in slots:
        tokens = int(rng.integers(1, max_blocks * page_size + 1))
        blocks = (tokens + page_size - 1) // page_size
        seq_tokens[slot] = tokens
        counts[slot] = blocks
        seq_blocks[slot, :blocks] = pool[cursor:cursor + blocks]
        cursor += blocks
    return seq_tokens, seq_blocks, counts, slots.astype(np.uint32)


def run_packing(torch, ops, row_slots, slot_active, seq_tokens, seq_blocks, rows, max_blocks, page_size, max_positions):
    capacity = seq_tokens.size
    positions = np.arange(max_positions, dtype=np.uint32)
    cos, sin = oracle.rope_rows(positions)
    rope_table = np.stack([cos, sin], axis=1)  # [position, 2, 64]
    u32 = lambda *shape: u32_out(torch, *shape)
    out = {
        "row_count": u32(1), "state_slots": u32(rows), "positions": u32(rows), "context_lengths": u32(rows),
        "physical_blocks": u32(rows), "block_offsets": u32(rows),
        "block_tables": u32_out(torch, rows, max_blocks, fill=7),
        "block_table_offsets": u32(rows + 1), "block_ids": u32(rows * max_blocks),
        "cosine": bf16_out(torch, rows, 64), "sine": bf16_out(torch, rows, 64), "status": u32(1),
    }
    ops.pack_decode_batch(None if row_slots is None else dev(torch, row_slots),
                          None if slot_active is None else dev(torch, slot_active), dev(torch, seq_tokens),
                          dev(torch, seq_blocks), dev(torch, rope_table), max_positions, out["row_count"],
                          out["state_slots"], out["positions"], out["context_lengths"], out["physical_blocks"],
                          out["block_offsets"], out["block_tables"], out["block_table_offsets"], out["block_ids"],
                          out["cosine"], out["sine"], out["status"], rows, capacity, max_blocks, page_size)
    torch.cuda.synchronize()
    return {k: host(v) for k, v in out.items()}, (cos, sin)


@pytest.mark.parametrize("page_size,capacity,live,max_blocks", [(16, 33, 32, 128), (64, 300, 257, 9), (16, 8, 1, 4)])
def test_pack_decode_batch_matches_host_layout_bit_for_bit(cuda, ops, page_size, capacity, live, max_blocks):
    seq_tokens, seq_blocks, counts, slots = packing_case(20, capacity, max_blocks, page_size, live)
    want = oracle.layout_decode(slots, seq_tokens, seq_blocks, counts, max_blocks, page_size)
    assert want["status"] == 0
    got, (cos, sin) = run_packing(cuda, ops, slots, None, seq_tokens, seq_blocks, live, max_blocks, page_size,
                                  max_blocks * page_size)
    assert got["status"][0] == 0 and got["row_count"][0] == live
    for key in ("state_slots", "positions", "context_lengths", "physical_blocks", "block_offsets", "block_tables",
                "block_table_offsets"):
        assert np.array_equal(got[key], want[key]), key
    total = int(want["block_table_offsets"][-1])
    assert np.array_equal(got["block_ids"][:total], want["block_ids"])
    want_cos, want_sin = oracle.rope_rows(want["positions"])
    assert np.array_equal(got["cosine"], want_cos) and np.array_equal(got["sine"], want_sin)


def test_pack_decode_batch_compacts_active_slots(cuda, ops):
    capacity, max_blocks, page_size = 700, 6, 16
    seq_tokens, seq_blocks, counts, slots = packing_case(21, capacity, max_blocks, page_size, 400)
    active = np.zeros(capacity, dtype=np.uint8)
    chosen = np.sort(slots[:333])
    active[chosen] = 1
    rows = 512  # capacity-level launch shape; the live prefix is reported on the device
    want = oracle.layout_decode(chosen, seq_tokens, seq_blocks, counts, max_blocks, page_size)
    got, _ = run_packing(cuda, ops, None, active, seq_tokens, seq_blocks, rows, max_blocks, page_size,
                         max_blocks * page_size)
    assert got["status"][0] == 0 and got["row_count"][0] == 333
    for key in ("state_slots", "positions", "context_lengths", "physical_blocks", "block_offsets"):
        assert np.array_equal(got[key][:333], want[key]), key
        assert not got[key][333:].any(), key
    assert np.array_equal(got["block_tables"][:333], want["block_tables"])
    assert not got["block_tables"][333:].any()
    assert np.array_equal(got["block_table_offsets"][:334], want["block_table_offsets"])
    assert np.all(got["block_table_offsets"][334:] == want["block_table_offsets"][-1])


def test_pack_decode_batch_reports_errors(cuda, ops):
    capacity, max_blocks, page_size = 10, 4, 16
    seq_tokens, seq_blocks, counts, slots = packing_case(22, capacity, max_blocks, page_size, 6)
    empty = [s for s in range(capacity) if seq_tokens[s] == 0][0]
    duplicate = np.array([slots[0], slots[1], slots[0]], dtype=np.uint32)
    for rows_in, code in [(np.array([slots[0], empty], dtype=np.uint32), 1), (duplicate, 2),
                          (np.array([99], dtype=np.uint32), 1)]:
        got, _ = run_packing(cuda, ops, rows_in, None, seq_tokens, seq_blocks, rows_in.size, max_blocks, page_size, 64)
        assert got["status"][0] == code
    too_long = seq_tokens.copy()
    too_long[slots[0]] = max_blocks * page_size + 1
    got, _ = run_packing(cuda, ops, slots[:1], None, too_long, seq_blocks, 1, max_blocks, page_size, 1000)
    assert got["status"][0] == 4


def test_page_table_apply_edits(cuda, ops):
    from qwencore_b200 import abi

    torch = cuda
    capacity, max_blocks = 5, 4
    seq_tokens = u32_out(torch, capacity)
    seq_blocks = u32_out(torch, capacity, max_blocks)
    edits = np.array([(2, 0, 9, 0), (2, 1, 4, 0), (2, 0, 17, 1), (3, 0, 5, 1), (3, 0, 1, 2), (7, 0, 1, 1)],
                     dtype=np.uint32)  # the last names a slot out of range and is ignored
    ops.page_table_apply(seq_tokens, seq_blocks, dev(torch, edits), len(edits), capacity, max_blocks)
    torch.cuda.synchronize()
    assert host(seq_tokens).tolist() == [0, 0, 17, 6, 0]
    assert host(seq_blocks)[2].tolist() == [9, 4, 0, 0]
    assert abi.lib.qwc_page_table_apply(0, 0, 0, 1, capacity, max_blocks, 0) == abi.CUDA_ERROR_INVALID_VALUE


# ---------------------------------------------------------------------------------------
# NVFP4 projections with both operands in four bits (at most eight rows, large matrices)
# ---------------------------------------------------------------------------------------

@pytest.mark.parametrize("out_features,in_features,batch", [(5128, 4096, 1), (5120, 4096, 2), (5120, 4096, 3),
                                                            (1400, 17408, 5), (5120, 6144, 8), (34816, 1024, 7)])
@pytest.mark.parametrize("std", [1.0, 3000.0, 1e-3], ids=["unit", "large", "small"])
def test_four_bit_projection_matches_oracle(cuda, ops, out_features, in_features, batch, std):
    """Every padding of the activation rows, ragged last tiles, one and several K slices, block scales of
    either sign, blocks whose activations differ by nine orders of magnitude, f16's largest binade, and a NaN."""
    torch = cuda
    packed, scales, _ = synth.nvfp4_matrix(41, "four_bit", out_features, in_features)
    flip = synth.generator(41, "signs").random(scales.shape) < 0.02
    scales = np.where(flip, scales | 0x80, scales).astype(np.uint8)
    swizzled = synth.swizzle_block_scales(scales, out_features, in_features)
    values = synth.bf16_value(synth.normal_bf16(41, "four_bit.x", (batch, in_features), std=std)).copy()
    values[:, 5::64] *= 30.0
    values[:, 7::64] *= 1e-6
    values[:, 256:512] = 0.0
    x = synth.bf16_bits(np.clip(values, -65280.0, 65280.0))
    want = oracle.gemv_w4a16(packed, scales, 2.0, x, out_features, in_features, batch)
    linear = ops.Linear(dev(torch, packed), dev(torch, swizzled), 2.0, out_features, in_features)
    out = bf16_out(torch, batch, out_features)
    linear.forward_w4a16(dev(torch, x), out, batch)
    torch.cuda.synchronize()
    clean = host(out).copy()
    assert_rms_close(synth.bf16_value(clean), want, "four-bit projection")
    poisoned = x.copy()
    poisoned[batch - 1, 17] = 0x7FC0  # a NaN stays in its row
    linear.forward_w4a16(dev(torch, poisoned), out, batch)
    torch.cuda.synchronize()
    assert np.isnan(synth.bf16_value(host(out))[batch - 1]).all()
    assert np.array_equal(host(out)[: batch - 1], clean[: batch - 1])


def test_four_bit_projection_saturates_at_the_largest_f16(cuda, ops):
    """Rows with values beyond 65504, with an infinity of either sign, and an ordinary one: the infinities become
    65504 like the rest (only NaN poisons).  Bound: half a bf16 step, one rounding of the magnitudes per 64 features."""
    torch = cuda
    out_features, in_features = 5120, 4096
    packed, scales, swizzled = synth.nvfp4_matrix(47, "saturate", out_features, in_features)
    x = synth.normal_bf16(47, "x", (4, in_features))
    x[0, 3::97] = synth.bf16_bits(np.resize(np.array([1e6, -7e4, 65536.0, -3e38], dtype=np.float32), x[0, 3::97].size))
    x[1, 1000] = synth.bf16_bits(np.array([np.inf], dtype=np.float32))[0]
    x[2, 17] = synth.bf16_bits(np.array([-np.inf], dtype=np.float32))[0]
    exact = np.clip(synth.bf16_value(x).astype(np.float64), -65504.0, 65504.0)
    weights = dequantize(packed, scales)
    got, _ = run_gemv(torch, ops, packed, scales, swizzled, 1.0, x, out_features, in_features, 4)
    want = exact @ weights.T
    bound = 2.0 ** -8 * np.abs(want) + (in_features / 64) * 2.0 ** -24 * (np.abs(exact) @ np.abs(weights).T)
    assert np.all(np.abs(got - want) <= bound)


def test_four_bit_swiglu_matches_oracle(cuda, ops):
    torch = cuda
    out_features, in_features, batch = 3336, 5120, 6
    gate, gate_scales, gate_swizzled = synth.nvfp4_matrix(42, "gate", out_features, in_features)
    up, up_scales, up_swizzled = synth.nvfp4_matrix(42, "up", out_features, in_features)
    x = synth.normal_bf16(42, "swiglu.x", (batch, in_features))
    want = oracle.swiglu_combine(oracle.gemv_w4a16(gate, gate_scales, 10.0, x, out_features, in_features, batch),
                                 oracle.gemv_w4a16(up, up_scales, 12.0, x, out_features, in_features, batch))
    out = bf16_out(torch, batch, out_features)
    ops.swiglu_w4a16(ops.Linear(dev(torch, gate), dev(torch, gate_swizzled), 10.0, out_features, in_features),
                     ops.Linear(dev(torch, up), dev(torch, up_swizzled), 12.0, out_features, in_features),
                     dev(torch, x), out, batch)
    torch.cuda.synchronize()
    assert_rms_close(synth.bf16_value(host(out)), want, "four-bit SwiGLU")


def dequantize(packed, scales):
    values = np.array([0, 0.5, 1, 1.5, 2, 3, 4, 6, 0, -0.5, -1, -1.5, -2, -3, -4, -6])
    codes = np.stack([packed & 15, packed >> 4], axis=-1).reshape(packed.shape[0], -1)
    return values[codes] * np.repeat(synth.e4m3_decode(scales).astype(np.float64), 16, axis=1)


@pytest.mark.parametrize("out_features,in_features", [(5120, 6144), (34816, 1024)], ids=["k_slices", "one_slice"])
@pytest.mark.parametrize("batch", [1, 2, 3, 4, 5, 8])
def test_four_bit_projection_keeps_small_activations_beside_large(cuda, ops, out_features, in_features, batch):
    """Every block of sixteen holds one large activation (up to f16's largest binade) where the weights are 0,
    and small ones elsewhere: the outputs are sums of the small ones alone, which f16 operands hold exactly.
    Bound: half a bf16 step of the result, and one rounding of 2^-24 of the magnitudes per 64 features."""
    torch = cuda
    rng = synth.generator(43, f"beside.{out_features}.{batch}")
    packed, scales, _ = synth.nvfp4_matrix(43, "beside", out_features, in_features)
    packed[:, 2::8] &= 0x0F  # feature 5 of every block
    swizzled = synth.swizzle_block_scales(scales, out_features, in_features)
    small = rng.uniform(0.002, 0.004, (batch, in_features)) * 2.0 ** rng.integers(-4, 3, (batch, in_features))
    values = (small * rng.choice([-1.0, 1.0], small.shape)).astype(np.float32)
    values[:, 5::16] = rng.choice([4096.0, -30000.0, 59904.0, -65280.0, 65504.0], (batch, in_features // 16))
    x = synth.bf16_bits(values)
    x[:, 0::64] = synth.bf16_bits(np.zeros((batch, in_features // 64), dtype=np.float32))
    exact = synth.bf16_value(x).astype(np.float64)
    exact[:, 5::16] = 0.0
    weights = dequantize(packed, scales)
    want = exact @ weights.T
    magnitudes = np.abs(exact) @ np.abs(weights).T
    got, _ = run_gemv(torch, ops, packed, scales, swizzled, 1.0, x, out_features, in_features, batch)
    bound = 2.0 ** -8 * np.abs(want) + (in_features / 64) * 2.0 ** -24 * magnitudes
    assert np.all(np.abs(got - want) <= bound)


@pytest.mark.parametrize("in_features", [6144, 17408])
def test_four_bit_projection_rounds_no_more_than_the_f16_kernel(cuda, ops, in_features):
    """Every block of sixteen features is there twice with opposite weights, shuffled over K: the exact result is
    0, and a call returns its own rounding.  Nine rows run on the f16 kernel, eight of them in four bits."""
    torch = cuda
    out_features, blocks = 5120, in_features // 16
    packed, scales, _ = synth.nvfp4_matrix(46, "rounding", out_features, in_features // 2)
    order = synth.generator(46, "order").permutation(blocks)
    packed = packed.reshape(out_features, blocks // 2, 8)
    packed = np.concatenate([packed, packed ^ 0x88], axis=1)[:, order].reshape(out_features, in_features // 2)
    scales = np.ascontiguousarray(np.concatenate([scales, scales], axis=1)[:, order])
    x = synth.normal_bf16(46, "x", (9, blocks // 2, 16))
    x = np.ascontiguousarray(np.concatenate([x, x], axis=1)[:, order].reshape(9, in_features))
    swizzled = synth.swizzle_block_scales(scales, out_features, in_features)
    four, _ = run_gemv(torch, ops, packed, scales, swizzled, 1.0, x[:8], out_features, in_features, 8)
    wide, _ = run_gemv(torch, ops, packed, scales, swizzled, 1.0, x, out_features, in_features, 9)
    assert np.any(four != 0) and np.sqrt(np.mean(np.square(four))) <= np.sqrt(np.mean(np.square(wide[:8])))


def test_four_bit_swiglu_divides_like_the_other_kernels(cuda, ops):
    """gate values around -88: 1 + exp(88) is beyond 2^126, where a fast division gives 0 instead of the quotient."""
    torch = cuda
    out_features, in_features, batch = 4096, 4096, 2
    gate = np.full((out_features, in_features // 2), 0x22, dtype=np.uint8)  # 1.0 everywhere
    scales = np.full((out_features, in_features // 16), 0x38, dtype=np.uint8)
    swizzled = synth.swizzle_block_scales(scales, out_features, in_features)
    x = synth.bf16_bits(np.stack([np.full(in_features, -88.0 / 4096, dtype=np.float32),
                                  np.full(in_features, -87.5 / 4096, dtype=np.float32)]))
    linear = ops.Linear(dev(torch, gate), dev(torch, swizzled), 1.0, out_features, in_features)
    up = ops.Linear(dev(torch, gate), dev(torch, swizzled), 2.0 ** -20, out_features, in_features)
    out = bf16_out(torch, batch, out_features)
    ops.swiglu_w4a16(linear, up, dev(torch, x), out, batch)
    torch.cuda.synchronize()
    value = synth.bf16_value(x).astype(np.float64).sum(-1)
    want = value / (1.0 + np.exp(-value)) * value * 2.0 ** 20
    got = synth.bf16_value(host(out)).astype(np.float64)
    # exp of fp32 arguments near 88: 88 * 2^-24 of the argument's rounding, and a bf16 result
    assert np.all(np.abs(got - want[:, None]) <= 0.01 * np.abs(want)[:, None])


@pytest.mark.parametrize("batch", [1, 8])
@pytest.mark.parametrize("kind", ["matrix", "pair", "head"])
def test_four_bit_projection_with_a_hint_stores_the_same_bytes(cuda, ops, batch, kind):
    """A K split (a cluster) and a whole K that name what follows: a large matrix, a pair, a vocabulary head."""
    torch = cuda
    from qwencore_b200 import abi
    x = dev(torch, synth.normal_bf16(44, "x", (batch, 5120)))

    def linear(name, out_features, in_features):
        packed, _, swizzled = synth.nvfp4_matrix(44, name, out_features, in_features)
        return ops.Linear(dev(torch, packed), dev(torch, swizzled), 8.0, out_features, in_features)

    after, after_up = linear("after", 5120, 6144), linear("after_up", 5120, 6144)
    table = torch.zeros((16384, 5120), dtype=torch.uint8, device="cuda")
    for out_features in (5128, 34816):
        now = linear("now", out_features, 5120)
        plain, hinted = bf16_out(torch, batch, out_features), bf16_out(torch, batch, out_features)
        now.forward_w4a16(x, plain, batch)
        if kind == "head":
            assert abi.lib.qwc_nvfp4_prefetch_next(table.data_ptr(), None, None, None, 16384, 5120, 2) == 0
        else:
            ops.prefetch_next(after, after_up if kind == "pair" else None)
        now.forward_w4a16(x, hinted, batch)
        torch.cuda.synchronize()
        assert np.array_equal(host(hinted), host(plain))
    assert abi.lib.qwc_device_status() == 0


@pytest.mark.parametrize("out_features,in_features", [(5120, 6144), (34816, 1024)], ids=["k_slices", "one_slice"])
@pytest.mark.parametrize("swiglu", [False, True], ids=["plain", "swiglu"])
def test_four_bit_projection_stores_nothing_once_a_wait_has_given_up(cuda, ops, out_features, in_features, swiglu):
    """With the status word set (as an earlier kernel leaves it), as the other projection kernels do."""
    torch = cuda
    from qwencore_b200 import abi
    packed, _, swizzled = synth.nvfp4_matrix(45, "status", out_features, in_features)
    linear = ops.Linear(dev(torch, packed), dev(torch, swizzled), 8.0, out_features, in_features)
    x = dev(torch, synth.normal_bf16(45, "x", (3, in_features)))
    out = dev(torch, np.full((3, out_features), 0x1234, dtype=np.uint16))
    torch.cuda.synchronize()
    assert abi.lib.qwc_device_status_set(0x103) == 0
    try:
        if swiglu:
            ops.swiglu_w4a16(linear, linear, x, out, 3)
        else:
            linear.forward_w4a16(x, out, 3)
        torch.cuda.synchronize()
        assert abi.lib.qwc_device_status() == 0x103
        assert np.all(host(out) == 0x1234)
    finally:
        assert abi.lib.qwc_device_status_reset() == 0
    linear.forward_w4a16(x, out, 3)
    torch.cuda.synchronize()
    assert np.isfinite(synth.bf16_value(host(out))).all()
