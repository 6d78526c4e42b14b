"""The host-side choices between kernels and launch shapes (pure functions of sizes; no GPU)."""
import os

import pytest
import torch

from ferrox_b200.kernels import ops
from ferrox_b200.parts.moe import expert_tile_tokens


def test_decode_split_plan_depends_on_sizes_only_and_stays_in_bounds():
    for tokens in (1, 2, 3, 8, 16, 33, 64, 200):
        for kv_blocks in (1, 4, 16, 28):
            for ctx in (64, 500, 4096, 32768):
                split_len, n = ops.decode_split_plan(tokens, kv_blocks, ctx)
                assert split_len == 0 and 1 <= n <= ops.DECODE_MAX_SPLITS
                assert n <= max(1, -(-ctx // 64))          # no run shorter than one tile of keys
                assert (split_len, n) == ops.decode_split_plan(tokens, kv_blocks, ctx)
    # 8 tokens x 16 kv heads: two runs fill one wave (256 of 444 blocks); a third adds no bandwidth
    assert ops.decode_split_plan(8, 16, 4096) == (0, 2)
    # the kernel that holds two blocks an SM and writes a single run's result itself
    assert ops.decode_split_plan(8, 16, 4096, 2, single_is_final=True) == (0, 2)
    assert ops.decode_split_plan(16, 16, 4096, 2, single_is_final=True) == (0, 1)
    assert ops.decode_split_plan(64, 16, 4096, 2, single_is_final=True) == (0, 1)
    # a single request: many runs, but no more than fill the machine
    assert 8 <= ops.decode_split_plan(1, 16, 4096)[1] <= ops.DECODE_MAX_SPLITS
    assert 8 <= ops.decode_split_plan(1, 16, 4096, 2, single_is_final=True)[1] <= ops.DECODE_MAX_SPLITS
    # many requests already fill the machine
    assert ops.decode_split_plan(200, 16, 4096)[1] <= 2


def test_which_product_kernel_takes_which_sizes():
    # few tokens against a big matrix: swapped roles only where measured faster
    assert not ops.swap_better(8, 6144, 2048) and ops.swap_better(40, 6144, 2048)
    assert ops.swap_better(8, 151936, 2048) and not ops.swap_better(4, 151936, 2048)
    assert not ops.swap_better(64, 2048, 5632)              # few rows of W: too few tiles
    # plain dense products of few tokens: runs of K so that 150 to 300 CTAs stream the matrix
    assert ops.swap_k_splits(64, 2048, 2048) == 8 and ops.swap_k_splits(64, 2048, 5632) == 8
    assert ops.swap_k_splits(64, 6144, 2048) == 4 and ops.swap_k_splits(8, 2048, 2048) == 0
    assert ops.swap_k_splits(32, 2048, 5632) > 0 and ops.swap_k_splits(32, 2048, 2048) == 0
    assert ops.swap_k_splits(64, 2048, 256) == 1      # never more runs than K allows
    # pairs of SMs need two rounds of 256 x 256 tiles for 74 pairs
    assert ops.pairs_better(2048, 6144) and not ops.pairs_better(2048, 2048) and not ops.pairs_better(512, 6144)
    assert ops.pairs_better(2048, 5632, gated=True)


def test_expert_tile_tokens_by_rows_per_expert():
    assert expert_tile_tokens(8, 4, 60) == (32, 32)
    assert expert_tile_tokens(64, 4, 60) == (32, 32)
    assert expert_tile_tokens(200, 4, 60) == (64, 64)
    assert expert_tile_tokens(2048, 4, 60) is None
    assert expert_tile_tokens(16, 8, 10) == (64, 64)       # few experts: more rows each


def test_decode_attention_by_tma_where_pages_and_heads_fit_its_boxes():
    import torch

    bf, f32 = torch.bfloat16, torch.float32
    # head sizes in steps of 64 on pages of a multiple of 64 positions, bfloat16 only
    assert ops.decode_tma_blocks_per_sm(bf, 128, 64) == 2 and ops.decode_tma_blocks_per_sm(bf, 64, 128) == 2
    assert ops.decode_tma_blocks_per_sm(bf, 256, 64) == 1 and ops.decode_tma_blocks_per_sm(bf, 192, 64) == 1
    for dtype, d, ps in ((f32, 128, 64), (bf, 96, 64), (bf, 128, 16), (bf, 128, 96), (bf, 320, 64), (bf, 0, 64)):
        assert ops.decode_tma_blocks_per_sm(dtype, d, ps) == 0


def test_routing_in_one_block_only_for_small_steps():
    assert ops.ROUTE_SMALL_MAX_TOKENS <= 64      # the one-block kernel takes a token per warp and round
    assert 32 * ops.ROUTE_SMALL_MAX_EXPERTS * 4 + (2 * ops.ROUTE_SMALL_MAX_EXPERTS + 1) * 4 <= 48 * 1024   # its shared memory


def test_prompt_attention_items_cover_every_key_block_once():
    """The planner of the tcgen05 prompt attention: every tile's key blocks are covered exactly once by its items, in
    order; a tile that was cut has consecutive parts and one merge row; heavy items come first; the cut depends on the
    step's sizes alone."""
    import random

    rng = random.Random(0)
    for trial in range(60):
        entries = [(rng.randint(1, 3000), rng.choice([0, 0, 5, 127, 128, 1000, 4097])) for _ in range(rng.randint(1, 4))]
        window = rng.choice([0, 0, 1, 100, 2048])
        heads = rng.choice([1, 16, 28])
        run_blocks = rng.choice([-1, -1, 0, 1, 2, 5])
        items, merges, parts = ops.prefill_tc_plan(entries, window, heads, run_blocks=run_blocks)
        again = ops.prefill_tc_plan(entries, window, heads, run_blocks=run_blocks)
        assert (items == again[0]).all() and (merges == again[1]).all() and parts == again[2]
        lengths = [int(it[5] - it[4]) for it in items]
        assert lengths == sorted(lengths, reverse=True) and min(lengths) >= 1
        by_tile = {}
        for tok0, rows, b, pos0, kb, ke, part, _ in items.tolist():
            by_tile.setdefault((tok0, rows, b, pos0), []).append((kb, ke, part))
        flat, n_tiles = 0, 0
        for b, (n, start) in enumerate(entries):
            for i in range(0, n, 256):
                rows, pos0 = min(256, n - i), start + i
                runs = sorted(by_tile[(flat + i, rows, b, pos0)])
                first = (max(0, pos0 - window + 1) if window else 0) // 128
                end = (pos0 + rows - 1) // 128 + 1
                assert runs[0][0] == first and runs[-1][1] == end
                assert all(a[1] == c[0] for a, c in zip(runs, runs[1:]))            # no gap, no overlap
                if len(runs) == 1:
                    assert runs[0][2] == -1
                else:
                    ps = [r[2] for r in runs]
                    assert ps == list(range(ps[0], ps[0] + len(runs))) and len(runs) <= ops.PREFILL_MAX_RUNS
                    assert [flat + i, rows, ps[0], len(runs)] in merges.tolist()
                n_tiles += 1
            flat += n
        assert len(by_tile) == n_tiles and parts == sum(m[3] for m in merges.tolist())
    # a prompt of 2,048 tokens on 16 heads: 128 whole tiles fit the 148 SMs at once; cutting would cost more than it saves
    items, merges, parts = ops.prefill_tc_plan([(2048, 0)], None, 16, sms=148)
    assert len(items) == 8 and parts == 0 and len(merges) == 0
    # a portion of 256 tokens behind 6,000 cached positions: one tile with 49 key blocks, cut so that all SMs work
    items, merges, parts = ops.prefill_tc_plan([(256, 6000)], None, 16, sms=148)
    assert parts == len(items) >= 6 and merges.tolist() == [[0, 256, 0, parts]]
    assert max(int(it[5] - it[4]) for it in items) <= 8
    # forced runs of four key blocks
    items, merges, parts = ops.prefill_tc_plan([(2048, 0)], None, 16, sms=148, run_blocks=4)
    assert len(items) == 20 and max(int(it[5] - it[4]) for it in items) == 4 and len(merges) == 6


def test_uploads_on_a_stream_beside_the_step_are_complete_when_they_return(monkeypatch):
    """A work list that a mixer beside the step's stream uploads is found by the others in ``batch.shared``, on streams that do
    not wait for that one: there the upload waits for its copy.  On the step's own stream it does not."""
    import numpy as np
    import torch

    waits = []

    class Stream:
        def synchronize(self):
            waits.append("copied" if copied else "too early")

    copied = []
    monkeypatch.setattr(ops, "_copied_behind", lambda t, device: copied.append(t) or t)      # (no device here)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda device=None: Stream())
    values = np.arange(4, dtype=np.int32)
    ops.upload(values, "cuda:0")
    with ops.stream_scope(11):
        ops.upload(values, "cuda:0")
        assert not waits
        with ops.stream_scope(22):
            ops.upload(values, "cuda:0")
            with ops.stream_scope(11):
                ops.upload(values, "cuda:0")
        assert waits == ["copied", "copied"]
        ops.upload(values, "cuda:0")
    ops.upload(values, "cuda:0")
    assert len(waits) == 2


def test_shared_memory_limits_are_not_asked_for_on_one_device_only():
    """The limit belongs to a function on the device that is current: an answer kept from the process's first call (which may
    also have been an error that passed) says nothing of a second device."""
    import os
    import re

    from ferrox_b200.kernels import lib

    for name in lib.sources():
        with open(os.path.join(lib.CSRC, name)) as f:
            assert not re.search(r"static\s+(const\s+)?\w+\s+\w+\s*=\s*cudaFuncSetAttribute", f.read()), name


def test_32_bit_product_plans_by_size():
    """Up to 4 rows the weights are streamed; beyond, tiles, in runs of K where they are few, whose partial sums stay within the
    workspace's limit; grids stay within their limits."""
    assert ops.F32_WORKSPACE_MAX <= 128 << 20
    assert [ops.gemm_f32_plan(m, 6144, 2048) for m in (1, 2, 3, 4)] == [(-1, 1), (-2, 1), (-4, 1), (-4, 1)]
    for m in (5, 16, 60, 129, 412, 517, 597, 2048, 2780, 70000, 3000000):
        for n in (1, 61, 2048, 15616, 151936):
            for k in (4, 128, 2048, 16384):
                form, splits = ops.gemm_f32_plan(m, n, k)
                assert form in (-8, 32, 64, 128) and 1 <= splits <= 16 and (form > 0 or splits == 1)
                assert splits == 1 or (4 * splits * m * n <= ops.F32_WORKSPACE_MAX and splits * 128 <= k)
                assert form < 0 or -(-m // form) <= 65535
    # groups: 2 or 4 rows a pass, from 65 rows on with a second kernel beside it, tiles above 6 rows a group
    assert [ops.gemm_f32_plan(m, 2816, 2048, 60) for m in (8, 60, 64, 65, 360, 361)] == [
        (-2, 1), (-2, 1), (-4, 1), (-4, 2), (-4, 2), (32, 1)]
    assert ops.gemm_f32_plan(100, 2816, 2048, 128) == (-2, 2) and ops.gemm_f32_plan(3000, 64, 64, 1025) == (32, 1)
    assert ops.gemm_f32_plan(60, 2048, 5632)[1] > 1 and ops.gemm_f32_plan(517, 15616, 2048)[1] > 1


def test_which_steps_take_a_recurrence_in_chunks():
    """Decisions where the two forms were measured more than a tenth apart."""
    from ferrox_b200.parts.linear_state import chunks_better

    for kind in ("delta", "mlstm", "general"):
        assert not chunks_better(kind, [31], 16, 128, 128) and not chunks_better(kind, [1] * 16 + [40], 16, 128, 128)
        for heads, d in ((2, 64), (4, 32), (16, 128), (32, 64), (64, 128), (64, 64)):
            assert chunks_better(kind, [2048], heads, d, d) and chunks_better(kind, [512], heads, d, d) or (kind, heads) == ("delta", 64)
        assert chunks_better(kind, [64], 2, 64, 64) and chunks_better(kind, [128], 16, 128, 128)
    # many short entries: a state is read and written for every chunk
    assert not chunks_better("delta", [32] * 16, 4, 128, 128) and not chunks_better("delta", [32] * 16, 64, 128, 128)
    assert not chunks_better("general", [32] * 16, 4, 128, 128) and not chunks_better("general", [32] * 16, 64, 64, 64)
    assert chunks_better("mlstm", [32] * 16, 16, 128, 128) and chunks_better("mlstm", [500] * 4, 64, 128, 128)
    assert chunks_better("delta", [500] * 4, 64, 128, 128) and chunks_better("delta", [500] * 4, 64, 64, 64)


def test_what_the_delta_rule_needs_first_by_runs_of_tokens_or_a_token_a_block(monkeypatch):
    """Runs of tokens take prompts from 128 tokens on, 32-bit rows on the 16-byte grid, heads of 64 and 128, four taps; the rest,
    and steps that move the tail on, a block a token."""
    import torch

    called = []
    monkeypatch.setattr(ops, "call", lambda name, *args: called.append(name))
    monkeypatch.setattr(ops, "_ptr", lambda t: 0)      # (no device here)

    def kernel(T=128, G=2, D=64, H=2, V=64, taps=4, cols=0, at=0, dtype=torch.float32, **more):
        C = 2 * G * D + H * V
        proj = torch.empty(T, C + cols + at, dtype=dtype)[:, at:]
        rows = lambda n: torch.empty(T, n)
        ops.delta_prep(proj, torch.empty(C, taps), taps, torch.empty(1, taps - 1, C), rows(2 * H), rows(1), rows(1),
                       torch.empty(T, dtype=torch.int32), torch.empty(1, dtype=torch.int32), rows(C), rows(H), rows(H), G, D, H, V,
                       stream=0, **more)
        return called.pop()

    for taken in (dict(), dict(T=3001), dict(D=128, G=1), dict(V=62), dict(cols=4), dict(H=3, V=4)):
        assert kernel(**taken) == "fx_delta_prep_runs", taken
    for refused in (dict(T=127), dict(T=1), dict(update_tail=True), dict(taps=3), dict(D=96), dict(G=1, D=32), dict(V=61), dict(cols=2),
                    dict(at=1, cols=3), dict(dtype=torch.bfloat16)):
        assert kernel(**refused) == "fx_delta_prep", refused


def test_32_bit_products_that_go_to_the_tensor_cores():
    """Many rows, 1,024 elements of K and more; workspaces within the limit; what the FFMA kernels are faster or nearer at stays."""
    assert [ops.gemm_f32_tc_tile(m, 15616, 2048) for m in (12, 64, 208, 209, 517)] == [16, 64, 208, 112, 176]
    assert ops.gemm_f32_tc_tile(517, 60, 2048) == 0 and ops.gemm_f32_tc_tile(517, 15616, 1020) == 0
    assert ops.gemm_f32_tc_tile(65, 257, 2048) == 0 and ops.gemm_f32_tc_tile(16, 2048, 2048) == 0
    for m in (9, 60, 209, 517, 2780, 70000):
        for n in (61, 2048, 151936):
            for k in (1024, 7808, 16384, 1 << 20):
                tile = ops.gemm_f32_tc_tile(m, n, k)
                assert tile % 16 == 0 and 0 <= tile <= ops.F32_TC_MAX_TILE
                if tile:
                    rows = min(m, ops._f32_tc_rows(k))
                    assert rows >= min(m, 208) and 6 * rows * k + 148 * 1024 * tile <= ops.F32_WORKSPACE_MAX


def test_tiles_of_dense_products_by_rounds():
    """Tiles that save a round of the SMs, narrow ones where the SMs are idle anyway, pairs where they need no more rounds."""
    assert [ops.dense_tile(m, 2048) for m in (96, 1531, 2048, 3001)] == [(False, 128), (False, 192), (False, 256), (False, 192)]
    assert [ops.dense_tile(m, 6144) for m in (517, 2048)] == [(False, 224), (True, 256)]
    assert ops.dense_tile(2600, 3584) == (False, 256) and ops.dense_tile(4096, 3584) == (True, 256) and ops.dense_tile(3000, 60) == (False, 128)
    for m in range(65, 5000, 97):
        for n in (512, 1000, 2048, 3584, 20480):
            pairs, tile = ops.dense_tile(m, n)
            assert tile in ((192, 256) if pairs else (128, 160, 192, 224, 256)) and (not pairs or ops.pairs_better(m, n))


def test_which_prompts_the_general_forms_take_to_tcgen05():
    """Where the two kernels were measured more than a tenth apart; kept blocks are an item's, of its first run only."""
    better = lambda e, window=None, heads=16, d=128, v=128, **k: ops.prefill_tc_better(e, window, heads, d, v, sms=148, **k)
    assert better([(2048, 0)], 1024, keep_first=4) and better([(256, 0)], 1024) and better([(16, 700)]) and better([(1531, 0)], d=192)
    assert better([(2048, 0)], 1024, capped=True) and better([(1531, 0)], heads=32, d=64, capped=True)
    assert not better([(9, 0)]) and not better([(40, 0)], capped=True)
    singles = [(1, 700)] * 15 + [(300, 0)]
    assert not better(singles, heads=32, d=64, capped=True) and not better(singles, 1024, capped=True)
    items, merges, parts = ops.prefill_tc_plan([(700, 0)], 150, 4, run_blocks=2, keep_first=200)
    for tok0, rows, entry, pos0, first, end, part, kept in items.tolist():
        blk = max(0, pos0 - 149) // 128
        assert kept == (min(2, blk) if first == blk else 0)
    assert all(k == 0 for *_, k in ops.prefill_tc_plan([(700, 0)], None, 4, keep_first=200)[0].tolist())


def test_walks_of_chunked_recurrences():
    """Longest entry first, each with its rows and its first chunk in the order of the batch."""
    assert ops.chunk_walks([33, 1, 100, 64]).tolist() == [[2, 34, 134, 3], [3, 134, 198, 7], [0, 0, 33, 0], [1, 33, 34, 2]]


def test_calls_by_the_extension_module_pass_what_ctypes_passes(tmp_path):
    """Every kind of argument, more integers and floats than registers hold, in mixed order; what is not read there is handed
    back; addresses and strides of tensors, and the errors of those that are none."""
    import ctypes
    import subprocess
    from ctypes import c_double, c_float, c_int, c_long, c_ulonglong, c_void_p

    from ferrox_b200.kernels import fastcall, hostlib

    if fastcall.module() is None:
        pytest.skip("no C compiler or no Python headers")
    kinds = [c_void_p, c_int, c_float, c_long, c_double, c_int, c_ulonglong, c_int, c_float, c_long, c_int, c_void_p, c_float, c_int,
             c_int, c_float, c_long, c_float, c_int, c_float, c_int, c_void_p, c_int, c_float, c_long]
    c_of = {c_void_p: "void*", c_int: "int", c_float: "float", c_long: "long", c_double: "double", c_ulonglong: "unsigned long long"}
    params = ", ".join(f"{c_of[k]} a{i}" for i, k in enumerate(kinds))
    store = " ".join(f"last[{i}] = (double){'(unsigned long)' if k is c_void_p else ''}a{i};" for i, k in enumerate(kinds))
    src = tmp_path / "f.cpp"
    src.write_text(f'extern "C" {{ static double last[99]; int f({params}) {{ {store} return -7; }} double get(int i) {{ return last[i]; }} }}')
    subprocess.run([hostlib._compiler(), "-O2", "-shared", "-fPIC", "-o", str(tmp_path / "f.so"), str(src)], check=True)
    lib = ctypes.CDLL(str(tmp_path / "f.so"))
    lib.f.argtypes, lib.f.restype, lib.get.restype = kinds, c_int, c_double
    value = {c_void_p: lambda i: None if i % 2 else 2 ** 47 + i, c_int: lambda i: -i if i % 3 else True, c_float: lambda i: i + 0.1,
             c_long: lambda i: -2 ** 40 - i, c_double: lambda i: i / 7, c_ulonglong: lambda i: 2 ** 63 + i}
    args = [value[k](i) for i, k in enumerate(kinds)]
    fast = fastcall.bind(lib.f, kinds)
    assert fast(*args) == -7
    got = [lib.get(i) for i in range(len(kinds))]
    assert lib.f(*args) == -7 and got == [lib.get(i) for i in range(len(kinds))]
    assert fast(ctypes.c_void_p(3), *args[1:]) is NotImplemented
    for bad in (args[:-1], args + [1], args[:2] + ["x"] + args[3:]):
        with pytest.raises(TypeError):
            fast(*bad)
    assert fastcall.bind(lib.f, [c_float] * 9) is None
    t = torch.zeros(3, 8)
    assert ops._ptr(None) is None and ops._rows(t[:, :5]) == 8
    for call in (lambda: ops._ptr(t), lambda: ops._rows(t.T), lambda: ops._rows(t[0])):
        with pytest.raises(ops.KernelError):
            call()


def test_work_of_the_32_bit_prompt_attention():
    """Each query is in one tile of one kernel, tiles hold no block that no query sees, and the planes' rows hold what they see."""
    for window in (None, 70, 200):
        for dim in (64, 128):
            entries = [(9, 0), (300, 0), (1, 700), (64, 0), (129, 63), (63, 0)]
            items, spans, rows, rest = ops.prefill_f32_tc_plan(entries, window, dim)
            taken = sorted((f, n, b, p) for f, n, b, p, *_ in items.tolist()) + sorted(map(tuple, rest.tolist()))
            seen = sorted(f + i for f, n, *_ in taken for i in range(n))
            assert seen == list(range(sum(n for n, _ in entries)))
            least = 64 if dim > 64 else 128
            assert {b for _, _, b, _ in taken[:len(items)]} == {b for b, (n, s) in enumerate(entries) if min(n + s, window or 9999) >= least}
            starts = [sum(n for n, _ in entries[:b]) for b in range(len(entries))]
            at = {b: (p0, end, row) for b, p0, end, row in spans.tolist()}
            for f, n, b, pos, lo, hi, row0, _ in items.tolist():
                assert f - starts[b] + entries[b][1] == pos and n <= ops.F32_TC_TILE
                p0, end, row = at[b]
                assert lo == ops.first_key(pos, window) // 64 and (hi - 1) * 64 <= pos + n - 1 < hi * 64
                assert row0 == row - p0 and p0 <= lo * 64 and row % 64 == 0 and row0 + hi * 64 <= rows
            assert [it[5] - it[4] for it in items.tolist()] == sorted((it[5] - it[4] for it in items.tolist()), reverse=True)
    assert ops.prefill_f32_tc_fits(3, 517, 576, 16, 16, 128) and not ops.prefill_f32_tc_fits(0, 9, 0, 16, 16, 128)
    assert not ops.prefill_f32_tc_fits(40, 5000, 5056, 16, 16, 128)


def test_decode_split_plan_of_the_32_bit_kernel():
    """Runs of whole 64 keys, in as few rounds of two blocks an SM as their length makes up for."""
    for tokens in (1, 3, 8, 64, 2000):
        for kv_blocks in (1, 4, 28):
            for ctx in (16, 64, 500, 4096, 65536):
                _, n = ops.decode_split_plan_f32(tokens, kv_blocks, ctx)
                assert 1 <= n <= min(ops.DECODE_F32_MAX_SPLITS, -(-ctx // 64))
    assert [ops.decode_split_plan_f32(t, 4, c)[1] for t, c in ((8, 2048), (4, 704), (1, 2048), (400, 2048))] == [8, 11, 32, 2]


def test_an_extension_module_that_does_not_build_or_load_leaves_the_calls_to_ctypes(tmp_path, monkeypatch):
    """A file that is no library in the module's place, a compiler that does not run: no module, now and when asked again; an import
    of the wrappers asks for none; an answer that the extension hands back is ctypes' one."""
    import subprocess
    import sys
    import sysconfig

    from ferrox_b200.kernels import fastcall

    monkeypatch.setattr(fastcall, "_module", None)
    monkeypatch.setattr(fastcall, "build_dir", lambda: str(tmp_path))
    path = fastcall.build()
    if path is None:
        pytest.skip("no C compiler or no Python headers")
    with open(path, "wb") as f:
        f.write(b"no library")
    assert fastcall.module() is None and fastcall.module() is None and fastcall.bind(None, []) is None
    tool = tmp_path / "cc"
    tool.write_text("not to be run")
    tool.chmod(0o600)
    monkeypatch.setattr(fastcall, "_module", None)
    monkeypatch.setattr(fastcall, "FLAGS", [*fastcall.FLAGS, "-DOTHER"])
    monkeypatch.setenv("CC", str(tool))
    assert fastcall.module() is None

    code = "import ferrox_b200.kernels.fastcall as f; f.build = lambda: 1 / 0; import ferrox_b200, ferrox_b200.kernels.ops"
    subprocess.run([sys.executable, "-c", code], check=True, cwd=os.path.dirname(os.path.dirname(os.path.abspath(__file__))))

    monkeypatch.setitem(ops._fast, "fx_none", lambda *a: NotImplemented)
    monkeypatch.setitem(ops._fn, "fx_none", lambda *a: 0)
    assert ops._answer("fx_none", 3) == 0

    # a module of another interpreter build is another file
    real = sysconfig.get_config_var
    monkeypatch.delenv("CC")
    names = set()
    for suffix in (".a.so", ".b.so"):
        monkeypatch.setattr(sysconfig, "get_config_var", lambda n, suffix=suffix: suffix if n == "EXT_SUFFIX" else real(n))
        names.add(fastcall.build())
    assert len(names) == 2


def test_shared_memory_limits_are_asked_for_without_a_flag():
    """No launcher remembers in a static that it has asked (the second device of a process would be refused at the launch)."""
    import re

    from ferrox_b200.kernels import lib

    for name in lib.sources():
        with open(os.path.join(lib.CSRC, name)) as f:
            text = f.read()
        for m in re.finditer(r"cudaFuncSetAttribute", text):
            before = text[max(0, m.start() - 300):m.start()]
            assert not re.search(r"static\s+(bool|int|size_t)\s+\w+\s*=\s*(false|0)\s*;", before), name
