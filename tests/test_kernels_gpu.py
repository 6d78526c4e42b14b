"""Each kernel alone against a plain 32-bit torch statement of the same operation,
at sizes other than the engine's (odd widths, head sizes in steps of 16, page
edges, windows)."""
import math
import random

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda:0"
DT = {"float32": torch.float32, "bfloat16": torch.bfloat16}
# error relative to the largest |expected| value
TOL = {"float32": 3e-6, "bfloat16": 1.2e-2}


def ops():
    from ferrox_b200.kernels import ops as o

    return o


def rel(got, want):
    return float((got.float() - want.float()).abs().max() / want.float().abs().max().clamp_min(1e-30))


def rnd(*shape, dtype=torch.float32, scale=1.0, seed=None):
    g = torch.Generator().manual_seed(seed if seed is not None else sum(shape) + len(shape))
    return (torch.randn(*shape, generator=g) * scale).to(dtype).to(DEV)


# ------------------------------------------------------------------ matrix products
@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("M,N,K", [(1, 7, 5), (3, 130, 77), (70, 65, 64), (129, 33, 250), (64, 64, 16)])
def test_gemm_generic(dtype, M, N, K):
    o, dt = ops(), DT[dtype]
    a, w, bias = rnd(M, K, dtype=dt), rnd(N, K, dtype=dt), rnd(N, dtype=torch.float32)
    want = a.float() @ w.float().T + bias
    out = torch.empty(M, N, dtype=dt, device=DEV)
    o.gemm(a, w, out, bias=bias)
    assert rel(out, want) < TOL[dtype]
    acc = rnd(M, N, dtype=torch.float32, seed=5)
    base = acc.clone()
    o.gemm(a, w, acc, accumulate=True)  # 32-bit output, added to what is there
    assert rel(acc, base + a.float() @ w.float().T) < (3e-6 if dtype == "float32" else 1e-5)


# sums of K products in another order: each is off by at most K roundings, in practice by about sqrt(K) of them
F32_FORMS = [(-1, 1), (-2, 1), (-4, 1), (-8, 1), (32, 1), (64, 1), (128, 1), (32, 3), (64, 2), (128, 5)]


@pytest.mark.parametrize("form,splits", F32_FORMS)
@pytest.mark.parametrize("M,N,K", [(1, 1, 4), (5, 61, 128), (9, 130, 1028), (33, 127, 20), (65, 257, 2048), (129, 128, 132)])
def test_gemm_f32_forms(form, splits, M, N, K, monkeypatch):
    """Both kernels of the 32-bit product at the edges of their tiles, passes and runs of K: with a bias, added to what
    is there, rows wider than K, and their error against 64-bit sums no larger than that of the same sums in order."""
    o = ops()
    monkeypatch.setattr(o, "gemm_f32_plan", lambda *a: (form, splits))
    a, w, bias = rnd(M, K + 4)[:, :K], rnd(N, K + 8)[:, :K], rnd(N)
    want = a.double() @ w.double().T
    out = torch.full((M, N + 3), 7.0, device=DEV)
    o.gemm(a, w, out[:, :N], bias=bias)
    assert rel(out[:, :N], want + bias) < 3e-6 and bool((out[:, N:] == 7).all())
    acc = rnd(M, N, seed=5)
    base = acc.clone()
    o.gemm(a, w, acc, accumulate=True)
    assert rel(acc, base + want) < 3e-6


@pytest.mark.parametrize("M,N,K,tile", [(1, 1, 4, 16), (16, 128, 32, 16), (17, 129, 36, 32), (40, 61, 132, 48), (81, 300, 1028, 96),
                                        (208, 257, 516, 208), (209, 2048, 2048, 112), (517, 130, 7808, 176), (130, 19000, 100, 144)])
def test_gemm_f32_on_tensor_cores(M, N, K, tile, monkeypatch):
    """The 32-bit product in three parts at the edges of its tiles, stages and shares of K: with a bias, added to what is there,
    rows wider than K.  Against 64-bit sums: what the parts leave out (2^-24 of a product) and a chain of K / 32 additions."""
    o = ops()
    monkeypatch.setattr(o, "gemm_f32_tc_tile", lambda *a: tile)
    monkeypatch.setattr(o, "gemm_f32_plan", lambda *a: (32, 1))
    a, w, bias = rnd(M, K + 4)[:, :K], rnd(N, K + 8)[:, :K], rnd(N)
    want = a.double() @ w.double().T
    out = torch.full((M, N + 3), 7.0, device=DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    o.gemm(a, w, out[:, :N], bias=bias, status=status)
    assert rel(out[:, :N], want + bias) < 5e-7 and bool((out[:, N:] == 7).all()) and int(status) == 0
    acc = rnd(M, N, seed=5)
    base = acc.clone()
    o.gemm(a, w, acc, accumulate=True)
    assert rel(acc, base + want) < 5e-7


def test_gemm_f32_on_tensor_cores_in_slices_of_rows(monkeypatch):
    o = ops()
    monkeypatch.setattr(o, "_f32_tc_rows", lambda k: 100)
    a, w = rnd(250, 1024), rnd(300, 1024)
    out = torch.empty(250, 300, device=DEV)
    o._gemm_f32_tc(a, w, out, 96, None, False, None, None)
    assert rel(out, a.double() @ w.double().T) < 5e-7


@pytest.mark.parametrize("cut", [False, True])
def test_gemm_f32_on_tensor_cores_beyond_finite_numbers(cut, monkeypatch):
    """Infinite operands, no numbers, overflows and small values: what the FFMA kernels give."""
    o = ops()
    monkeypatch.setattr(o, "gemm_f32_plan", lambda *a: (32, 1))
    M, N, K = 20, 128 * (5 if cut else 148), 256
    a, w = rnd(M, K), rnd(N, K)
    a[3, 200], a[4, 7], a[5] = float("inf"), float("nan"), 0.0
    a[6:8] = 0.0         # (one product each: where sums overflow on the way depends on their order)
    a[6, 10], a[7, 0] = 3e38, torch.finfo(torch.float32).max
    a[8] *= 1e-30
    w[9, 100], w[10, 5], w[11, 2] = float("-inf"), float("nan"), 0.0
    w[12] *= 1e-3
    a[9, 64] = float("inf")
    w[9, 65] = float("inf")
    want, out = torch.empty(M, N, device=DEV), torch.empty(M, N, device=DEV)
    monkeypatch.setattr(o, "gemm_f32_tc_tile", lambda *x: 0)
    o.gemm(a, w, want)
    monkeypatch.setattr(o, "gemm_f32_tc_tile", lambda *x: 32)
    o.gemm(a, w, out)
    assert bool(((out == want) | (out.isnan() == want.isnan()))[~want.isfinite()].all())
    assert torch.equal(out.isfinite(), want.isfinite()) and torch.equal(out[out.isinf()], want[want.isinf()])
    ok = want.isfinite()
    exact, size = a.double() @ w.double().T, a.double().abs() @ w.double().abs().T
    assert bool(((out.double() - exact).abs() <= 2e-6 * size)[ok].all())


def test_gemm_f32_on_tensor_cores_single_products(monkeypatch):
    """Results of one product each, some of operands whose lower parts are as large as they can be: what the parts leave out is up to
    2^-24 of it, and the accumulator's cut up to one unit in the last place."""
    o = ops()
    M, N, K = 100, 300, 1024
    a, w, at = torch.zeros(M, K, device=DEV), rnd(N, K), torch.arange(M, device=DEV)
    a[at, at * 7] = rnd(M, 1)[:, 0]
    largest = (torch.arange(M, device=DEV, dtype=torch.int32) + 0x3f808000 - M).view(torch.float32)      # 1 + 2^-8 less a few units
    a[M // 2:, :] = 0
    a[at[M // 2:], at[M // 2:] * 7] = largest[M // 2:]
    w[N // 2:, :] = largest[torch.arange(N - N // 2, device=DEV) % M][:, None]
    out, want = torch.empty(M, N, device=DEV), a.double() @ w.double().T
    monkeypatch.setattr(o, "gemm_f32_plan", lambda *x: (32, 1))
    monkeypatch.setattr(o, "gemm_f32_tc_tile", lambda *x: 112)
    o.gemm(a, w, out)
    assert float(((out.double() - want) / want).abs().max()) <= 1.5 * 2 ** -23
    # the same where cut parts would have the most to leave out, 1 + 2^-7 less a few units
    a[a != 0], w[:] = 1 + 2 ** -7 - 2 ** -22, 1 + 2 ** -7 - 2 ** -21
    want = a.double() @ w.double().T
    o.gemm(a, w, out)
    assert float(((out.double() - want) / want).abs().max()) <= 1.5 * 2 ** -23


def test_gemm_f32_on_tensor_cores_below_the_parts_range(monkeypatch):
    """Operands whose second and third parts are subnormal or nothing, against weights that make the results large: what is lost of an
    operand is below 2^-133."""
    o = ops()
    M, N, K = 60, 200, 1024
    a, w = rnd(M, K) * torch.tensor([1e-33, 1e-35, 1e-36, 1e-37, 1e-38], device=DEV).repeat(M // 5)[:, None], rnd(N, K) * 1e30
    out, size = torch.empty(M, N, device=DEV), w.double().abs()
    monkeypatch.setattr(o, "gemm_f32_plan", lambda *x: (32, 1))
    monkeypatch.setattr(o, "gemm_f32_tc_tile", lambda *x: 64)
    o.gemm(a, w, out)
    err = (out.double() - a.double() @ w.double().T).abs()
    assert bool((err <= 2.0 ** -133 * size.sum(1) + 2e-6 * (a.double().abs() @ size.T)).all())


@pytest.mark.parametrize("M,N,K", [(64, 3072, 2048), (517, 2048, 7808)])
def test_gemm_f32_on_tensor_cores_sums_of_one_sign(M, N, K, monkeypatch):
    """Operands of one sign, where every cut of the accumulator has that sign too: two cuts of a stage's sum by up to a unit in its last
    place, half of it on average (2^-24 to 2^-23 of the result), and the roundings of a chain of K / 32 sums; at most twice as far
    from 64 bits as the FFMA kernel."""
    o = ops()
    a, w = rnd(M, K).abs(), rnd(N, K).abs()
    want, off = a.double() @ w.double().T, {}
    tile = o.gemm_f32_tc_tile(M, N, K)
    assert tile
    for t in (tile, 0):
        monkeypatch.setattr(o, "gemm_f32_tc_tile", lambda *x, t=t: t)
        out = torch.empty(M, N, device=DEV)
        o.gemm(a, w, out)
        off[bool(t)] = float((out.double() - want).norm() / want.norm())
    assert off[True] < 2 ** -22 and off[True] < 2 * off[False], off


@pytest.mark.parametrize("form", [-1, -4, -8, 32, 64, 128])
def test_gemm_f32_groups(form, monkeypatch):
    """Groups without rows, of one row, of a tile's rows and one more, with gathered rows, more groups than a warp."""
    o = ops()
    monkeypatch.setattr(o, "gemm_f32_plan", lambda *a: (form, 1))
    G, N, K, T = 40, 130, 68, 50
    x, w = rnd(T, K), rnd(G, N, K)
    counts = [0] * G
    for g, c in ((1, 1), (2, 32), (5, 33), (31, 9), (32, 64), (33, 129), (39, 2)):
        counts[g] = c
    off = [0]
    for c in counts:
        off.append(off[-1] + c)
    rows = torch.randint(0, T, (off[-1],), generator=torch.Generator().manual_seed(1)).to(torch.int32).to(DEV)
    offsets = torch.tensor(off, dtype=torch.int32, device=DEV)
    want = torch.cat([x[rows[off[g]:off[g + 1]].long()].double() @ w[g].double().T for g in range(G)])
    out = torch.empty(off[-1], N, device=DEV)
    o.gemm(x, w, out, a_rows=rows, group_offsets=offsets)
    assert rel(out, want) < 3e-6


@pytest.mark.parametrize("counts,tiles", [([6] * 40, False), ([1] * 39 + [100], False), ([0] * 39 + [240], True),
                                          ([0] * 17 + [60, 60, 60, 60] + [0] * 19, True), ([0] * 40, False)])
def test_gemm_f32_groups_go_by_their_sizes(counts, tiles, monkeypatch):
    """Up to 6 rows a group on average: weights streamed, unless a few groups have most rows; the results are those of the one
    kernel or of the other, bit for bit, and all there."""
    o = ops()
    M, G, N, K = 240, len(counts), 2048, 2048
    w = torch.randn(G, N, K, device=DEV, generator=torch.Generator(device=DEV).manual_seed(1))
    x, off = rnd(M, K), [0]
    for c in counts:
        off.append(off[-1] + c)
    offsets = torch.tensor(off, dtype=torch.int32, device=DEV)
    out = torch.full((M, N), 3.0, device=DEV)
    o.gemm(x, w, out, group_offsets=offsets)
    plan = o.gemm_f32_plan(M, N, K, G)
    alone = {}
    for name, form in (("stream", plan[0]), ("tiles", 32)):
        monkeypatch.setattr(o, "gemm_f32_plan", lambda *a: (form, 1))
        alone[name] = torch.full((M, N), 3.0, device=DEV)
        o.gemm(x, w, alone[name], group_offsets=offsets)
    assert torch.equal(out, alone["tiles" if tiles else "stream"])
    if off[-1]:
        assert not torch.equal(alone["tiles"], alone["stream"])
        want = torch.cat([x[off[g]:off[g + 1]].double() @ w[g].double().T for g in range(G)])
        assert rel(out[:off[-1]], want) < 3e-6
    assert bool((out[off[-1]:] == 3).all())


def test_gemm_mixed_precision_weights_stay_32_bit():
    o = ops()
    a, w = rnd(5, 96, dtype=torch.bfloat16), rnd(40, 96, dtype=torch.float32)
    out = torch.empty(5, 40, dtype=torch.float32, device=DEV)
    o.gemm(a, w, out)
    assert rel(out, a.float() @ w.T) < 3e-6  # no rounding of the 32-bit weights


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_gemm_grouped_with_gather(dtype):
    o, dt = ops(), DT[dtype]
    G, N, K, T = 5, 37, 48, 23
    x, w = rnd(T, K, dtype=dt), rnd(G, N, K, dtype=dt)
    counts = [0, 9, 1, 0, 13]
    offsets = torch.tensor([0] + list(torch.tensor(counts).cumsum(0)), dtype=torch.int32, device=DEV)
    rows = torch.randint(0, T, (sum(counts),), generator=torch.Generator().manual_seed(1)).to(torch.int32).to(DEV)
    out = torch.zeros(sum(counts), N, dtype=dt, device=DEV)
    o.gemm(x, w, out, a_rows=rows, group_offsets=offsets)
    r = 0
    for g, c in enumerate(counts):
        for _ in range(c):
            want = x[rows[r]].float() @ w[g].float().T
            assert rel(out[r], want) < TOL[dtype]
            r += 1


@pytest.mark.parametrize("T", [1, 3, 8, 9, 17, 40, 64])
@pytest.mark.parametrize("N,K", [(16, 32), (60, 64), (1, 96), (200, 2048), (33, 160), (9493, 64)])
def test_gemm_skinny(T, N, K):
    o = ops()
    x, w, bias = rnd(T, K, dtype=torch.bfloat16), rnd(N, K, dtype=torch.bfloat16, scale=0.1), rnd(N)
    want = x.float() @ w.float().T + bias
    out = torch.empty(T, N, dtype=torch.bfloat16, device=DEV)
    o.gemm_skinny(x, w, out, bias=bias)
    assert rel(out, want) < TOL["bfloat16"]
    acc = rnd(T, N, seed=3)
    base = acc.clone()
    o.gemm_skinny(x, w, acc, accumulate=True)
    assert rel(acc, base + x.float() @ w.float().T) < 2e-5
    # gated: silu(gate) * up in the epilogue
    if N > 1:
        wg = rnd(2 * N, K, dtype=torch.bfloat16, scale=0.1, seed=9)
        gate, up = x.float() @ wg[:N].float().T, x.float() @ wg[N:].float().T
        got = torch.empty(T, N, dtype=torch.float32, device=DEV)
        o.gemm_skinny(x, wg, got, gated=True)
        assert rel(got, gate / (1 + torch.exp(-gate)) * up) < 2e-5


@pytest.mark.parametrize("T", [1, 5, 8, 13, 32])
@pytest.mark.parametrize("N,K", [(6144, 2048), (1000, 384), (2048, 2048), (61, 128), (7, 1408), (3001, 1024)])
def test_gemm_slab_holds_its_rows_of_the_matrix_in_shared_memory(T, N, K):
    """The product for a few tokens that asks for the whole matrix before it waits for the kernel before it:
    against the 32-bit product, with a bias, added to a 32-bit result, rows of x wider than K, after a kernel
    that is still running when it starts (the same stream: its wait is what orders them)."""
    o = ops()
    xw = rnd(T, K + 24, dtype=torch.bfloat16)
    x = xw[:, :K]
    w, bias = rnd(N, K, dtype=torch.bfloat16, scale=0.1), rnd(N)
    assert o.slab_ok(x, w)
    want = x.float() @ w.float().T
    out = torch.empty(T, N, dtype=torch.bfloat16, device=DEV)
    o.gemm_slab(x, w, out, bias=bias)
    assert rel(out, want + bias) < TOL["bfloat16"]
    acc = rnd(T, N, seed=3)
    base = acc.clone()
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    o.gemm_slab(x, w, acc, accumulate=True, status=status)
    assert rel(acc, base + want) < 2e-5 and int(status) == 0
    # x written by the kernel just before it on the stream
    x2 = torch.empty_like(xw)
    out2 = torch.empty(T, N, dtype=torch.float32, device=DEV)
    o.residual_add(acc, out)                      # some kernel of the library: the product's wait is for it
    x2.copy_(xw)
    o.gemm_slab(x2[:, :K], w, out2)
    assert rel(out2, want) < 2e-5
    # each token's result does not depend on the others
    if T > 1:
        one = torch.empty(1, N, dtype=torch.float32, device=DEV)
        o.gemm_slab(x[T - 1:T], w, one)
        assert torch.equal(one[0], out2[T - 1])


def test_gemm_slab_refuses_what_does_not_fit():
    o = ops()
    big = torch.empty(40000, 2048, dtype=torch.bfloat16, device=DEV)      # 164 MB: no SM's share fits
    x = rnd(4, 2048, dtype=torch.bfloat16)
    assert not o.slab_ok(x, big)
    assert not o.slab_ok(rnd(4, 96, dtype=torch.bfloat16), rnd(64, 96, dtype=torch.bfloat16))      # K no multiple of 128
    assert not o.slab_ok(rnd(40, 128, dtype=torch.bfloat16), rnd(64, 128, dtype=torch.bfloat16))   # too many tokens
    assert not o.slab_ok(rnd(4, 128), rnd(64, 128))                                                  # 32-bit
    with pytest.raises(o.KernelError):
        o.gemm_slab(x, big, torch.empty(4, 40000, dtype=torch.float32, device=DEV))


@pytest.mark.parametrize("T,K_top", [(1, 2), (8, 4), (33, 3)])
def test_gemm_skinny_grouped_against_routing(T, K_top):
    o = ops()
    E, I, H = 7, 64, 96
    x = rnd(T, H, dtype=torch.bfloat16)
    w_gu, w_down = rnd(E, 2 * I, H, dtype=torch.bfloat16, scale=0.1), rnd(E, H, I, dtype=torch.bfloat16, scale=0.1)
    g = torch.Generator().manual_seed(T)
    ids = torch.stack([torch.randperm(E, generator=g)[:K_top] for _ in range(T)]).to(torch.int32).to(DEV)
    scratch = torch.zeros(2 * E, dtype=torch.int32, device=DEV)
    offsets = torch.empty(E + 1, dtype=torch.int32, device=DEV)
    src = torch.empty(T * K_top, dtype=torch.int32, device=DEV)
    inv = torch.empty(T * K_top, dtype=torch.int32, device=DEV)
    active = torch.empty(min(E, T * K_top), dtype=torch.int32, device=DEV)
    o.moe_align(ids, E, scratch, offsets, src, inv, active)
    # bookkeeping: a permutation, rows grouped by expert, active = experts with rows
    counts = torch.bincount(ids.flatten().long(), minlength=E)
    assert offsets.tolist() == [0] + counts.cumsum(0).tolist()
    assert sorted(inv.tolist()) == list(range(T * K_top))
    for i in range(T * K_top):
        r = int(inv[i])
        e = int(ids.flatten()[i])
        assert int(offsets[e]) <= r < int(offsets[e + 1]) and int(src[r]) == i // K_top
    act_list = [e for e in active.tolist() if e >= 0]
    assert act_list == [e for e in range(E) if counts[e] > 0] and all(e == -1 for e in active.tolist()[len(act_list):])
    act = torch.empty(T * K_top, I, dtype=torch.bfloat16, device=DEV)
    o.gemm_skinny(x, w_gu, act, gated=True, x_rows=src, group_offsets=offsets, active_groups=active, tokens_hint=T)
    y = torch.empty(T * K_top, H, dtype=torch.float32, device=DEV)
    o.gemm_skinny(act, w_down, y, group_offsets=offsets, active_groups=active, tokens_hint=T)
    for i in range(T * K_top):
        t, e, r = i // K_top, int(ids.flatten()[i]), int(inv[i])
        gu = x[t].float() @ w_gu[e].float().T
        a = (gu[:I] / (1 + torch.exp(-gu[:I])) * gu[I:])
        assert rel(act[r], a) < TOL["bfloat16"]
        assert rel(y[r], act[r].float() @ w_down[e].float().T) < 2e-5


def test_skinny_refuses_what_it_cannot_do():
    o = ops()
    x, w = rnd(2, 40, dtype=torch.bfloat16), rnd(16, 40, dtype=torch.bfloat16)
    assert not o.skinny_ok(x, w)
    with pytest.raises(o.KernelError, match="size"):
        o.gemm_skinny(x, w, torch.empty(2, 16, dtype=torch.bfloat16, device=DEV))
    with pytest.raises(o.KernelError, match="CUDA tensors"):
        o.gemm(x.cpu(), w, torch.empty(2, 16, dtype=torch.bfloat16, device=DEV))


# ------------------------------------------------------------------ element-wise
@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("H", [16, 80, 333, 2048])
def test_rmsnorm_embed_silu(dtype, H):
    o, dt = ops(), DT[dtype]
    x, w = rnd(9, H, scale=3.0), rnd(H, dtype=dt) + 1
    eps = 1e-5
    want = x * (1.0 / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)) * w.float()
    out = torch.empty(9, H, dtype=dt, device=DEV)
    o.rmsnorm(x, w, eps, out)
    assert rel(out, want) < (1e-6 if dtype == "float32" else 5e-3)
    rows = torch.tensor([7, 0, 7, 3], dtype=torch.int32, device=DEV)
    picked = torch.empty(4, H, dtype=dt, device=DEV)
    o.rmsnorm(x, w, eps, picked, rows=rows)
    assert torch.equal(picked, out[rows.long()])
    table = rnd(50, H, dtype=dt)
    ids = torch.tensor([3, 49, 0, 3], dtype=torch.int32, device=DEV)
    h = torch.empty(4, H, dtype=torch.float32, device=DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    o.embed(table, ids, h, status)
    assert torch.equal(h, table[ids.long()].float()) and int(status) == 0
    o.embed(table, torch.tensor([50], dtype=torch.int32, device=DEV), h[:1], status)
    assert int(status) == 1  # a token id outside the table is reported, not read
    gu = rnd(5, 2 * H, dtype=dt)
    act = torch.empty(5, H, dtype=dt, device=DEV)
    o.silu_mul(gu, act)
    g, u = gu[:, :H].float(), gu[:, H:].float()
    assert rel(act, g / (1 + torch.exp(-g)) * u) < (1e-6 if dtype == "float32" else 5e-3)


def test_router_topk_and_ties():
    o = ops()
    logits = torch.arange(1.0, 9.0, device=DEV).reshape(1, 8)
    ids = torch.empty(1, 3, dtype=torch.int32, device=DEV)
    w = torch.empty(1, 3, dtype=torch.float32, device=DEV)
    o.router_topk(logits, 3, False, ids, w)
    assert ids.tolist() == [[7, 6, 5]]
    # the reference's golden for these logits (crates/ferrox-moe/src/lib.rs:864-893), its tolerance
    assert torch.allclose(w.cpu(), torch.tensor([[0.6323223, 0.2326232, 0.0855683]]), atol=1e-4)
    o.router_topk(logits, 3, True, ids, w)
    assert abs(float(w.sum()) - 1) < 1e-6
    tie = torch.tensor([[0.5, 2.0, 2.0, 0.1, 2.0]], device=DEV)
    ids2 = torch.empty(1, 2, dtype=torch.int32, device=DEV)
    o.router_topk(tie, 2, False, ids2, torch.empty(1, 2, device=DEV))
    assert ids2.tolist() == [[1, 2]]  # equal probabilities: the lowest index first
    g = torch.Generator().manual_seed(0)
    big = torch.randn(300, 61, generator=g).to(DEV)
    ids3 = torch.empty(300, 5, dtype=torch.int32, device=DEV)
    w3 = torch.empty(300, 5, device=DEV)
    o.router_topk(big, 5, False, ids3, w3)
    p = torch.softmax(big, -1)
    tv, ti = torch.topk(p, 5, dim=-1)
    assert torch.equal(ids3.long(), ti) and rel(w3, tv) < 1e-6


def test_moe_combine_in_rank_order():
    o = ops()
    T, K, H = 6, 3, 40
    y, shared = rnd(T * K, H), rnd(T, H)
    inv = torch.randperm(T * K, generator=torch.Generator().manual_seed(0)).to(torch.int32).to(DEV)
    w = torch.rand(T, K, generator=torch.Generator().manual_seed(1)).to(DEV)
    gate = rnd(T, 1)
    h = rnd(T, H, seed=2)
    want = h.clone()
    for t in range(T):
        acc = torch.zeros(H, device=DEV)
        for k in range(K):
            acc = acc + w[t, k] * y[inv[t * K + k]]
        want[t] += acc + torch.sigmoid(gate[t]) * shared[t]
    o.moe_combine(h, y, inv, w, shared, gate)
    assert rel(h, want) < 1e-6


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("H", [40, 2048, 3584, 8192, 1000])
@pytest.mark.parametrize("with_shared", [True, False])
def test_moe_combine_with_the_norm_that_follows(dtype, H, with_shared):
    """The combine that also applies the next RMSNorm: the same residual rows, bit for bit, as the combine alone, and
    the normed rows of the norm kernel on them (sums of squares in another order: a rounding apart)."""
    o, dt = ops(), DT[dtype]
    T, K = 5, 4
    y, shared = rnd(T * K, H, dtype=dt), (rnd(T, H, dtype=dt) if with_shared else None)
    inv = torch.randperm(T * K, generator=torch.Generator().manual_seed(0)).to(torch.int32).to(DEV)
    w = torch.rand(T, K, generator=torch.Generator().manual_seed(1)).to(DEV)
    logits = rnd(T, 7)
    gate = logits[:, 6:] if with_shared else None      # a strided column, as the router's product leaves it
    nw = (1 + 0.1 * rnd(H, seed=5)).to(dt)
    h0 = rnd(T, H, seed=2)
    h_a, h_b = h0.clone(), h0.clone()
    o.moe_combine(h_a, y, inv, w, shared, gate)
    x_a = o.rmsnorm(h_a, nw, 1e-5, torch.empty(T, H, dtype=dt, device=DEV))
    assert o.combine_norm_ok(h_b, y) == (H % (4 if dtype == "float32" else 8) == 0 and H // (4 if dtype == "float32" else 8) <= 1024)
    if not o.combine_norm_ok(h_b, y):
        return
    x_b = o.moe_combine(h_b, y, inv, w, shared, gate, norm=(nw, 1e-5, torch.empty(T, H, dtype=dt, device=DEV)))
    assert torch.equal(h_a, h_b)
    assert rel(x_b.float(), x_a.float()) < (1e-6 if dtype == "float32" else 8e-3)
    want = h_a / torch.sqrt((h_a * h_a).mean(dim=1, keepdim=True) + 1e-5) * nw.float()
    assert rel(x_b.float(), want) < (1e-6 if dtype == "float32" else 8e-3)


# ------------------------------------------------------------------ rotary + cache write + attention
def build_cache(dtype, seqs, nkv, d, page_size, n_pages, seed=0):
    """Random K/V for requests of the given lengths, scattered into shuffled pages."""
    rng = random.Random(seed)
    free = list(range(n_pages))
    rng.shuffle(free)
    width = max(-(-L // page_size) for L in seqs) + 1
    table = torch.full((len(seqs) + 2, width), -1, dtype=torch.int32)
    kp = torch.zeros(n_pages, nkv, page_size, d)
    vp = torch.zeros(n_pages, nkv, page_size, d)
    ks, vs = [], []
    for s, L in enumerate(seqs):
        k = torch.randn(L, nkv, d, generator=torch.Generator().manual_seed(seed * 100 + s)).to(dtype).float()
        v = torch.randn(L, nkv, d, generator=torch.Generator().manual_seed(seed * 100 + 50 + s)).to(dtype).float()
        ks.append(k)
        vs.append(v)
        for j in range(-(-L // page_size)):
            pg = free.pop()
            table[s + 1, j] = pg  # slot = s + 1: slots and entries are different things
            n = min(page_size, L - j * page_size)
            kp[pg, :, :n] = k[j * page_size:j * page_size + n].transpose(0, 1)
            vp[pg, :, :n] = v[j * page_size:j * page_size + n].transpose(0, 1)
    return kp.to(dtype).to(DEV), vp.to(dtype).to(DEV), table.to(DEV), ks, vs


def plain_attention(q, k, v, pos, window, scale):
    """One query (heads, d) at position pos over keys k[:pos+1] (nkv heads)."""
    nh, nkv = q.shape[0], k.shape[1]
    lo = max(0, pos - window + 1) if window else 0
    out = torch.zeros_like(q)
    for h in range(nh):
        kv = h // (nh // nkv)
        s = (k[lo:pos + 1, kv] @ q[h]) * scale
        out[h] = torch.softmax(s, 0) @ v[lo:pos + 1, kv]
    return out


ATT_CASES = [
    # nh, nkv, d, page, window, lengths
    (4, 2, 16, 4, 0, [1, 5, 33]),
    (2, 1, 64, 16, 16, [70, 16, 17]),
    (6, 3, 48, 8, 7, [40, 9]),
    (16, 16, 128, 64, 0, [300, 64, 65]),
    (28, 4, 128, 64, 100, [130]),
    (3, 3, 256, 16, 0, [50]),
    (12, 1, 32, 16, 0, [90]),
    # head sizes in steps of 64 on pages of a multiple of 64: in bfloat16 the decode kernel that streams pages by TMA
    (8, 2, 64, 64, 0, [200, 129, 1]),
    (6, 2, 192, 128, 150, [318, 70]),
    (40, 2, 64, 128, 0, [150, 260]),
    (4, 4, 256, 64, 33, [140, 64]),
    (16, 16, 128, 64, 70, [319]),
]


@pytest.mark.parametrize("case", [
    # nh, nkv, d, page, window, softcap, [(keys before the portion, tokens of the portion)]
    (4, 2, 16, 4, 0, None, [(0, 1), (0, 33), (63, 2)]),
    (6, 3, 48, 8, 7, 5.0, [(30, 40), (0, 9)]),
    (16, 16, 128, 64, 0, None, [(64, 65), (0, 64), (127, 1)]),
    (28, 4, 124, 128, 100, 30.0, [(200, 70)]),
    (3, 1, 68, 96, 0, None, [(95, 97)]),
])
def test_prefill_attention_f32(case):
    """The 32-bit tiled prompt attention against the plain statement, and, where a portion's last key and value are not
    numbers, every query before it as if they were not there."""
    o = ops()
    nh, nkv, d, ps, window, cap, portions = case
    lens = [a + n for a, n in portions]
    kp, vp, table, ks, vs = build_cache(torch.float32, lens, nkv, d, ps, n_pages=sum(-(-L // ps) for L in lens) + 3)
    T = sum(n for _, n in portions)
    q = rnd(T, nh * d + 8)
    tiles, flat = [], 0
    for b, (start, n) in enumerate(portions):
        tiles += [(flat + i, min(32, n - i), b, start + i) for i in range(0, n, 32)]
        flat += n
    tiles = torch.tensor(tiles, dtype=torch.int32, device=DEV)
    slots = torch.tensor([b + 1 for b in range(len(lens))], dtype=torch.int32, device=DEV)
    out = torch.empty(T, nh * d, device=DEV)
    assert o.prefill_f32_ok(q, out, kp, d)
    args = (table, ps, tiles, slots, out, nh, nkv, d, window, d ** -0.5)
    o.prefill_attention_f32(q, kp, vp, *args, softcap=cap)
    flat, last = 0, []
    for b, (start, n) in enumerate(portions):
        for i in range(n):
            pos, qi = start + i, q[flat + i, :nh * d].cpu().view(nh, d)
            lo = max(0, pos - window + 1) if window else 0
            for h in range(nh):
                s = (ks[b][lo:pos + 1, h * nkv // nh] @ qi[h]) * d ** -0.5
                s = cap * torch.tanh(s / cap) if cap else s
                want = torch.softmax(s, 0) @ vs[b][lo:pos + 1, h * nkv // nh]
                assert rel(out[flat + i].view(nh, d)[h].cpu(), want) < 5e-6
        flat += n
        last.append(flat - 1)
    before = out.clone()
    for b, L in enumerate(lens):
        page = int(table[b + 1, (L - 1) // ps])
        kp[page, :, (L - 1) % ps], vp[page, :, (L - 1) % ps] = float("nan"), float("inf")
    o.prefill_attention_f32(q, kp, vp, *args, softcap=cap)
    keep = [t for t in range(T) if t not in last]
    assert torch.equal(out[keep], before[keep])


@pytest.mark.parametrize("case", [
    # heads, kv heads, head_dim, page size, window, cap, [(first position, tokens)], an entry's page that is not there
    (4, 2, 128, 64, 0, None, [(0, 64), (0, 129), (500, 1), (63, 65)], None),
    (6, 3, 64, 128, 150, 5.0, [(0, 128), (777, 127), (127, 130), (0, 9)], None),
    (3, 1, 80, 64, 0, None, [(5, 300), (0, 33)], (0, 1)),
    (2, 2, 72, 64, 70, None, [(0, 400), (129, 1)], None),
])
def test_prefill_attention_f32_on_tensor_cores(case):
    """32-bit prompt attention from bfloat16 parts, short entries by the FFMA kernel, against 64 bits; then with keys and values that
    are no finite numbers, where it has to be none where the FFMA kernel's is none."""
    o = ops()
    nh, nkv, d, ps, window, cap, portions, hole = case
    lens = [a + n for a, n in portions]
    kp, vp, table, ks, vs = build_cache(torch.float32, lens, nkv, d, ps, n_pages=sum(-(-L // ps) for L in lens) + 3)
    T, scale = sum(n for _, n in portions), d ** -0.5
    q = rnd(T, nh * d + 8)
    slots = torch.tensor([b + 1 for b in range(len(lens))], dtype=torch.int32, device=DEV)
    if hole:
        table[hole[0] + 1, hole[1]] = -1
    items, spans, rows, rest = o.prefill_f32_tc_plan([(n, s) for s, n in portions], window, d)
    ffma, flat = [], 0
    for b, (start, n) in enumerate(portions):
        ffma += [(flat + i, min(32, n - i), b, start + i) for i in range(0, n, 32)]
        flat += n
    ffma = torch.tensor(ffma, dtype=torch.int32, device=DEV)
    items, spans, rest = (torch.from_numpy(x).to(DEV) for x in (items, spans, rest))
    out, plain, status = torch.empty(T, nh * d, device=DEV), torch.empty(T, nh * d, device=DEV), torch.zeros(1, dtype=torch.int32, device=DEV)
    assert o.prefill_f32_tc_ok(q, out, kp, ps, d) and items.shape[0] and not o.prefill_f32_tc_ok(q[:, 2:], out, kp, ps, d)

    def run():
        out.fill_(7.0)
        o.prefill_attention_f32_tc(q, kp, vp, table, ps, items, spans, rows, slots, out, nh, nkv, d, window, scale, status=status, softcap=cap)
        if rest.shape[0]:
            o.prefill_attention_f32(q, kp, vp, table, ps, rest, slots, out, nh, nkv, d, window, scale, softcap=cap)
        o.prefill_attention_f32(q, kp, vp, table, ps, ffma, slots, plain, nh, nkv, d, window, scale, softcap=cap)
        assert int(status) == 0

    run()
    flat, bound = 0, torch.empty(T, nh, 1)
    for b, (start, n) in enumerate(portions):
        pos, key = torch.arange(start, start + n)[:, None], torch.arange(start + n)
        sees = (key <= pos) & (key > pos - (window or 1 << 30))
        if hole and hole[0] == b:
            sees &= key // ps != hole[1]
        x = q[flat:flat + n, :nh * d].cpu().double().view(n, nh, d)
        k, v = (t[b].double().repeat_interleave(nh // nkv, 1) for t in (ks, vs))
        s = torch.einsum("thd,khd->htk", x, k) * scale
        s = cap * torch.tanh(s / cap) if cap else s
        want = torch.einsum("htk,khd->thd", torch.softmax(s.masked_fill(~sees, float("-inf")), -1), v)
        # A score's sum is cut once for each 16 elements (by a unit of at most |q| |k| in 24 bits), what the six products leave out is
        # a few units more, and expf, tanhf and the scale some; a weight is off by that and its sum's, and a block's result, by cuts of
        # the same kind, by a unit for each 16 keys.
        unit = 2.0 ** -23
        es = unit * (d / 16 + 8) * scale * x.norm(dim=-1).max() * k.norm(dim=-1).max()
        bound[flat:flat + n] = v.abs().max() * (2 * es + unit * (8 + (start + n) / 16))
        err = (out[flat:flat + n].cpu().double().view(n, nh, d) - want).abs()
        assert bool((err <= bound[flat:flat + n]).all()), float((err / bound[flat:flat + n]).max())
        flat += n
    before = out.clone()
    for b, L in enumerate(lens):
        page = int(table[b + 1, (L - 1) // ps])
        kp[page, :, (L - 1) % ps], vp[page, :, (L - 1) % ps] = float("nan"), float("inf")
    page = int(table[1, 0])                  # (the first entry sees these, where they are not out of its window)
    kp[page, 0, 3, 1], vp[page, 0, 5, 2], vp[page, 0, 6, 3] = float("inf"), float("-inf"), float("nan")
    run()
    assert torch.equal(out.isnan(), plain.isnan()) and torch.equal(out.isinf(), plain.isinf())
    fine = plain.isfinite()
    for seen, other in ((before, portions[0][1]), (plain, 0)):       # (the other entries as if they were not there, but for their last)
        off = (out - seen).abs().view(T, nh, d) <= 2 * bound.to(DEV)
        assert bool((off | ~fine.view(T, nh, d))[other:].all())


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("case", ATT_CASES)
@pytest.mark.parametrize("kernel", ["generic", "decode"])
def test_attention_over_pages(dtype, case, kernel):
    o, dt = ops(), DT[dtype]
    nh, nkv, d, ps, window, lens = case
    kp, vp, table, ks, vs = build_cache(dt, lens, nkv, d, ps, n_pages=sum(-(-L // ps) for L in lens) + 3)
    # queries: for each request its last position, one in the middle and position 0
    toks = []
    for s, L in enumerate(lens):
        for pos in sorted({L - 1, L // 2, 0}):
            toks.append((s, pos))
    T = len(toks)
    q = rnd(T, nh * d + 8, dtype=dt)[:, : nh * d + 8]  # rows wider than the heads: a strided view
    positions = torch.tensor([p for _, p in toks], dtype=torch.int32, device=DEV)
    token_seq = torch.tensor([s for s, _ in toks], dtype=torch.int32, device=DEV)
    seq_slot = torch.tensor([s + 1 for s in range(len(lens))], dtype=torch.int32, device=DEV)
    out = torch.empty(T, nh * d, dtype=dt, device=DEV)
    scale = 1 / math.sqrt(d)
    if kernel == "generic":
        o.paged_attention(q, kp, vp, table, ps, positions, token_seq, seq_slot, out, nh, nkv, d, window, scale)
    else:
        for split_len, n_splits in ((64, 5), (128, 3), (4096, 1), (0, 1), (0, 3), (0, 7)):
            pa = torch.empty(T, nh, n_splits, d, device=DEV)
            pm = torch.empty(T, nh, n_splits, 2, device=DEV)
            out.zero_()
            o.decode_attention(q, kp, vp, table, ps, positions, token_seq, seq_slot, out, nh, nkv, d, window, scale,
                               split_len, n_splits, pa, pm)
            _check_attention(out, q, ks, vs, toks, nh, d, window, scale, dtype)
            # the key ranges merged by the kernel's last blocks instead of the merge kernel: the same bits, twice
            # in a row with the same counters, which it leaves zeroed
            counters = torch.zeros(T * nkv * -(-(nh // nkv) // 16), dtype=torch.int32, device=DEV)
            for _ in range(2):
                fused = torch.zeros_like(out)
                o.decode_attention(q, kp, vp, table, ps, positions, token_seq, seq_slot, fused, nh, nkv, d, window,
                                   scale, split_len, n_splits, torch.empty_like(pa), torch.empty_like(pm),
                                   counters=counters)
                assert torch.equal(fused, out)
                assert int(counters.abs().sum()) == 0
        return
    _check_attention(out, q, ks, vs, toks, nh, d, window, scale, dtype)


@pytest.mark.parametrize("nh,nkv,d,ps,cap", [
    (4, 4, 8, 3, None), (6, 3, 32, 24, None), (8, 2, 64, 64, None), (5, 5, 64, 16, None), (16, 2, 60, 40, None), (4, 2, 128, 64, 9.0),
    (9, 9, 96, 7, None), (12, 3, 100, 64, None), (9, 1, 128, 64, None), (6, 3, 200, 48, None),
])
def test_decode_attention_f32_forms(nh, nkv, d, ps, cap):
    """The 32-bit decode kernel with each number of query heads and width of heads that it has a form for: runs that end in a tile,
    at its end and one past it, against 64 bits."""
    o = ops()
    lens = [1, 31, 32, 33, 64, 65, 129, 300]
    kp, vp, table, ks, vs = build_cache(torch.float32, lens, nkv, d, ps, n_pages=sum(-(-L // ps) for L in lens) + 3)
    T, scale = len(lens), d ** -0.5
    q, out = rnd(T, nh * d), torch.empty(T, nh * d, device=DEV)
    positions, token_seq, slots = (torch.tensor(x, dtype=torch.int32, device=DEV) for x in ([L - 1 for L in lens], range(T), range(1, T + 1)))
    for split_len, n_splits in ((0, 1), (0, 5), (16, 19), (33, 10)):
        pa, pm = torch.full((T, nh, n_splits, d), float("nan"), device=DEV), torch.full((T, nh, n_splits, 2), float("nan"), device=DEV)
        o.decode_attention(q, kp, vp, table, ps, positions, token_seq, slots, out, nh, nkv, d, None, scale, split_len, n_splits, pa, pm,
                           softcap=cap)
        for b, L in enumerate(lens):
            x = q[b].cpu().double().view(nh, d)
            k, v = (t[b].double().repeat_interleave(nh // nkv, 1) for t in (ks, vs))
            s = torch.einsum("hd,khd->hk", x, k) * scale
            s = cap * torch.tanh(s / cap) if cap else s
            want = torch.einsum("hk,khd->hd", torch.softmax(s, -1), v)
            # a sum of d products rounds d times by half a unit of at most |q| |k|, the weights and their sums by some units more
            unit = 2.0 ** -23
            es = unit * (d / 2 + 8) * scale * x.norm(dim=-1).max() * k.norm(dim=-1).max()
            assert float((out[b].cpu().double().view(nh, d) - want).abs().max()) <= v.abs().max() * (2 * es + unit * (8 + L / 2)), (b, n_splits)


def _check_attention(out, q, ks, vs, toks, nh, d, window, scale, dtype):
    for i, (s, pos) in enumerate(toks):
        want = plain_attention(q[i, : nh * d].float().cpu().reshape(nh, d), ks[s], vs[s], pos, window, scale)
        got = out[i].float().cpu().reshape(nh, d)
        assert rel(got, want) < (2e-6 if dtype == "float32" else 1e-2), (s, pos)


@pytest.mark.parametrize("kernel", ["generic", "decode"])
def test_attention_finds_one_far_key_and_respects_the_window_edge(kernel):
    """One key among hundreds is made to stand out; the output must be its value when
    it is visible and must not contain it one position past the window."""
    o = ops()
    nh = nkv = 2
    d, ps, L = 32, 16, 400
    kp, vp, table, ks, vs = build_cache(torch.float32, [L], nkv, d, ps, n_pages=30, seed=4)
    far = 37
    q = torch.zeros(1, nh * d)
    spike = torch.randn(d, generator=torch.Generator().manual_seed(1))
    spike = spike / spike.norm() * 12
    q[0, :d], q[0, d:] = spike, spike
    page, off = int(table[1, far // ps]), far % ps
    kp[page, :, off, :] = (spike * 8).to(DEV)  # score far above every other key
    ks[0][far, :, :] = spike * 8
    q = q.to(DEV)
    args = dict(n_heads=nh, n_kv_heads=nkv, head_dim=d, scale=1 / math.sqrt(d))
    positions = torch.tensor([L - 1], dtype=torch.int32, device=DEV)
    z = torch.zeros(1, dtype=torch.int32, device=DEV)
    slot = torch.ones(1, dtype=torch.int32, device=DEV)

    def run(window):
        out = torch.empty(1, nh * d, device=DEV)
        if kernel == "generic":
            o.paged_attention(q, kp, vp, table, ps, positions, z, slot, out, window=window, **args)
        else:
            pa, pm = torch.empty(1, nh, 7, d, device=DEV), torch.empty(1, nh, 7, 2, device=DEV)
            o.decode_attention(q, kp, vp, table, ps, positions, z, slot, out, window=window, split_len=64, n_splits=7,
                               part_acc=pa, part_ml=pm, **args)
        return out.cpu().reshape(nh, d)

    full = run(0)
    assert rel(full[0], vs[0][far, 0]) < 1e-4  # all the weight on the far key
    inside = run(L - far)  # window reaches back exactly to the far key
    assert rel(inside[0], vs[0][far, 0]) < 1e-4
    outside = run(L - far - 1)  # one less: the far key is out
    want = plain_attention(q[0].cpu().reshape(nh, d), ks[0], vs[0], L - 1, L - far - 1, args["scale"])
    assert rel(outside, want) < 1e-5 and rel(outside[0], vs[0][far, 0]) > 0.1


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("nh,nkv,d,rot", [(4, 2, 16, 16), (3, 1, 48, 48), (2, 2, 128, 64)])
def test_rope_and_cache_write(dtype, nh, nkv, d, rot):
    o, dt = ops(), DT[dtype]
    ps, T = 4, 7
    theta = 10000.0
    width = nh * d + 2 * nkv * d
    qkv = rnd(T, width, dtype=dt)
    before = qkv.clone()
    positions = torch.tensor([0, 1, 2, 3, 9, 10, 150], dtype=torch.int32, device=DEV)
    token_seq = torch.tensor([0, 0, 0, 0, 1, 1, 2], dtype=torch.int32, device=DEV)
    seq_slot = torch.tensor([2, 0, 1], dtype=torch.int32, device=DEV)
    table = torch.full((3, 40), -1, dtype=torch.int32)
    table[2, 0], table[0, 2], table[1, 37] = 5, 1, 3
    table = table.to(DEV)
    kp = torch.zeros(6, nkv, ps, d, dtype=dt, device=DEV)
    vp = torch.zeros_like(kp)
    inv_freq = (1.0 / torch.pow(torch.tensor(theta), torch.arange(0, rot // 2).float() * 2 / rot)).to(DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    o.rope_kv_write(qkv, positions, token_seq, seq_slot, inv_freq, rot, kp, vp, table, ps, nh, nkv, d, True, status)
    assert int(status) == 0
    x = before.float().cpu()
    ang = positions.cpu().float()[:, None] * inv_freq.cpu()[None, :]
    cos, sin = torch.cos(ang), torch.sin(ang)
    tol = 2e-6 if dtype == "float32" else 8e-3
    for t in range(T):
        for hh in range(nh + nkv):
            a, b = x[t, hh * d: hh * d + rot // 2], x[t, hh * d + rot // 2: hh * d + rot]
            want = torch.cat([a * cos[t] - b * sin[t], a * sin[t] + b * cos[t], x[t, hh * d + rot:(hh + 1) * d]])
            assert rel(qkv[t, hh * d:(hh + 1) * d].cpu(), want) < tol
        assert torch.equal(qkv[t, (nh + nkv) * d:], before[t, (nh + nkv) * d:])  # v untouched
    # where the rows landed: page table[slot][pos // ps], offset pos % ps
    where = {0: (5, 0), 1: (5, 1), 2: (5, 2), 3: (5, 3), 4: (1, 1), 5: (1, 2), 6: (3, 2)}
    for t, (pg, off) in where.items():
        assert torch.equal(kp[pg, :, off, :].reshape(-1), qkv[t, nh * d:(nh + nkv) * d])
        assert torch.equal(vp[pg, :, off, :].reshape(-1), qkv[t, (nh + nkv) * d:])
    assert int((kp != 0).any(dim=-1).sum()) == T * nkv  # nothing else was written
    # a position without a page is reported, not written
    o.rope_kv_write(qkv[:1], torch.tensor([20], dtype=torch.int32, device=DEV), token_seq[:1], seq_slot, inv_freq, rot,
                    kp, vp, table, ps, nh, nkv, d, True, status)
    assert int(status) == 2


@pytest.mark.parametrize("T,E,K", [(1, 4, 2), (8, 60, 4), (33, 61, 5), (256, 8, 3)])
def test_route_small_equals_the_two_step_routing(T, E, K):
    o = ops()
    logits = rnd(T, E, scale=2.0, seed=T)
    i32 = dict(dtype=torch.int32, device=DEV)
    ids_a, w_a = torch.empty(T, K, **i32), torch.empty(T, K, device=DEV)
    o.router_topk(logits, K, True, ids_a, w_a)
    ids_b, w_b = torch.empty(T, K, **i32), torch.empty(T, K, device=DEV)
    offsets, src, inv = torch.empty(E + 1, **i32), torch.empty(T * K, **i32), torch.empty(T * K, **i32)
    active = torch.empty(min(E, T * K), **i32)
    o.route_small(logits, K, True, ids_b, w_b, offsets, src, inv, active)
    assert torch.equal(ids_a, ids_b) and torch.equal(w_a, w_b)
    counts = torch.bincount(ids_b.flatten().long(), minlength=E)
    assert offsets.tolist() == [0] + counts.cumsum(0).tolist()
    assert sorted(inv.tolist()) == list(range(T * K))
    flat = ids_b.flatten().tolist()
    for i, r in enumerate(inv.tolist()):
        assert int(offsets[flat[i]]) <= r < int(offsets[flat[i] + 1]) and int(src[r]) == i // K
    act = [e for e in active.tolist() if e >= 0]
    assert act == [e for e in range(E) if counts[e] > 0]


@pytest.mark.parametrize("T,E,K", [(1, 4, 2), (70, 60, 4), (2048, 61, 5), (700, 1000, 8), (300, 8, 3)])
def test_route_in_two_kernels_equals_the_separate_steps(T, E, K):
    o = ops()
    logits = rnd(T, E + 1, scale=2.0, seed=T)      # one more column than experts, as with the shared expert's gate
    i32 = dict(dtype=torch.int32, device=DEV)
    ids_a, w_a = torch.empty(T, K, **i32), torch.empty(T, K, device=DEV)
    o.router_topk(logits, K, True, ids_a, w_a, n_experts=E)
    ids_b, w_b = torch.empty(T, K, **i32), torch.empty(T, K, device=DEV)
    offsets, src, inv = torch.empty(E + 1, **i32), torch.empty(T * K, **i32), torch.empty(T * K, **i32)
    active = torch.empty(min(E, T * K), **i32)
    scratch = torch.full((2 * E,), 7, **i32)       # the call clears it itself
    for _ in range(2):
        o.route(logits, K, True, ids_b, w_b, scratch, offsets, src, inv, active, n_experts=E)
        assert torch.equal(ids_a, ids_b) and torch.equal(w_a, w_b)
        counts = torch.bincount(ids_b.flatten().long(), minlength=E)
        assert offsets.tolist() == [0] + counts.cumsum(0).tolist()
        inv_l, src_l, off_l, flat = inv.tolist(), src.tolist(), offsets.tolist(), ids_b.flatten().tolist()
        assert sorted(inv_l) == list(range(T * K))
        assert all(off_l[flat[i]] <= r < off_l[flat[i] + 1] and src_l[r] == i // K for i, r in enumerate(inv_l))
        act = [e for e in active.tolist() if e >= 0]
        assert act == [e for e in range(E) if counts[e] > 0][: active.numel()]


def test_rope_table_matches_inline_angles():
    o = ops()
    nh, nkv, d, ps = 2, 1, 32, 8
    T = 5
    positions = torch.tensor([0, 3, 77, 1000, 4095], dtype=torch.int32, device=DEV)
    inv_freq = (1.0 / torch.pow(torch.tensor(1e6), torch.arange(0, d // 2).float() * 2 / d)).to(DEV)
    table = torch.empty(T, d // 2, 2, device=DEV)
    o.rope_table(positions, inv_freq, table)
    ang = positions.float()[:, None] * inv_freq[None, :]
    assert rel(table[..., 0], torch.cos(ang)) < 1e-6 and rel(table[..., 1], torch.sin(ang)) < 1e-6
    qkv = rnd(T, (nh + 2 * nkv) * d)
    a, b = qkv.clone(), qkv.clone()
    z = torch.zeros(T, dtype=torch.int32, device=DEV)
    slot = torch.zeros(1, dtype=torch.int32, device=DEV)
    bt = torch.arange(0, 520, dtype=torch.int32, device=DEV).reshape(1, -1)
    kp = torch.zeros(520, nkv, ps, d, device=DEV)
    vp = torch.zeros_like(kp)
    o.rope_kv_write(a, positions, z, slot, inv_freq, d, kp, vp, bt, ps, nh, nkv, d)
    o.rope_kv_write(b, positions, z, slot, inv_freq, d, kp, vp, bt, ps, nh, nkv, d, cos_sin=table)
    assert torch.equal(a, b)  # the table holds exactly the angles the kernel would compute


# ------------------------------------------------------------------ tcgen05 products
@pytest.mark.parametrize("M,N,K", [(128, 128, 64), (256, 384, 512), (65, 60, 72), (300, 200, 2048), (129, 130, 200),
                                   (2048, 256, 1408), (2048, 6144, 2048), (1000, 1000, 520), (4096, 640, 72)])
def test_gemm_tc_dense(M, N, K):
    o = ops()
    x, w, bias = rnd(M, K, dtype=torch.bfloat16), rnd(N, K, dtype=torch.bfloat16, scale=0.1), rnd(N)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    want = x.float() @ w.float().T
    out = torch.full((M, N), 7.0, dtype=torch.bfloat16, device=DEV)
    o.gemm_tc(x, w, out, bias=bias, status=status)
    assert int(status) == 0
    assert rel(out, want + bias) < TOL["bfloat16"]
    acc = rnd(M, N, seed=3)
    base = acc.clone()
    o.gemm_tc(x, w, acc, accumulate=True, status=status)
    assert int(status) == 0 and rel(acc, base + want) < 2e-5
    # a strided view of wider rows, as the attention output is inside the fused q|k|v rows
    wide = rnd(M, K + 64, dtype=torch.bfloat16, seed=11)
    out32 = torch.empty(M, N, dtype=torch.float32, device=DEV)
    o.gemm_tc(wide[:, :K], w, out32, status=status)
    assert rel(out32, wide[:, :K].float() @ w.float().T) < 2e-5


@pytest.mark.parametrize("pairs,tile", [(False, 160), (False, 192), (False, 224), (True, 192)])
@pytest.mark.parametrize("M,N,K", [(65, 64, 72), (129, 512, 136), (300, 1344, 2048), (1000, 1001, 520)])
def test_dense_tiles_of_other_widths(pairs, tile, M, N, K):
    """Tiles narrower than 256 rows of w, whose last 32 columns may have no partner to fill a line with: bit for bit what the
    widest tiles give (each element's sum runs over K in one order), with a bias, in both types, added to what is there."""
    o = ops()
    x, w, bias = rnd(M, K, dtype=torch.bfloat16), rnd(N, K, dtype=torch.bfloat16, scale=0.1), rnd(N)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    kern = o.gemm_tc2 if pairs else o.gemm_tc
    for dt, acc in ((torch.bfloat16, False), (torch.float32, False), (torch.float32, True)):
        got, want = (torch.full((M, N + 8), 7.0, dtype=dt, device=DEV) for _ in range(2))
        for t, out in ((tile, got), (256, want)):
            kern(x, w, out[:, :N], bias=bias, accumulate=acc, tile=t, status=status)
        assert int(status) == 0 and torch.equal(got, want) and bool((got[:, N:] == 7).all())
        assert rel(got[:, :N], x.float() @ w.float().T + bias + (7 if acc else 0)) < (TOL["bfloat16"] if dt == torch.bfloat16 else 2e-5)


@pytest.mark.parametrize("M,N,K", [(256, 256, 64), (300, 520, 136), (2048, 2048, 2048), (70, 100, 96), (1000, 6144, 264)])
def test_gemm_tc2_pairs_of_sms(M, N, K):
    """The dense product on pairs of SMs (cta_group::2): plain with bias, accumulating, into a strided view."""
    o = ops()
    x, w = rnd(M, K, dtype=torch.bfloat16), rnd(N, K, dtype=torch.bfloat16, scale=0.2)
    bias = rnd(N, seed=5)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    want = x.float() @ w.float().T
    out = torch.full((M, N), 7.0, dtype=torch.bfloat16, device=DEV)
    o.gemm_tc2(x, w, out, bias=bias, status=status)
    assert int(status) == 0
    assert rel(out, want + bias) < TOL["bfloat16"]
    acc = rnd(M, N, seed=3)
    base = acc.clone()
    o.gemm_tc2(x, w, acc, accumulate=True, status=status)
    assert int(status) == 0 and rel(acc, base + want) < 2e-5
    wide = torch.full((M, N + 5), 7.0, device=DEV)
    o.gemm_tc2(x, w, wide[:, :N], status=status)
    assert rel(wide[:, :N], want) < 2e-5 and float(wide[:, N:].min()) == 7.0


@pytest.mark.parametrize("M,N,K", [(1, 60, 64), (8, 200, 96), (33, 4100, 136), (64, 2048, 512), (70, 100, 96),
                                   (300, 520, 136), (2048, 2048, 264)])
def test_products_with_the_squared_relu_in_their_epilogue(M, N, K):
    """Every product kernel that takes an activation on its result, the kernel ``linear`` picks, and ``linear`` where
    the picked kernel has no epilogue for it (runs of K): relu(x w^T + b)^2, which the plain product and the plain
    ReLU both miss by far."""
    o = ops()
    x, w, bias = rnd(M, K, dtype=torch.bfloat16), rnd(N, K, dtype=torch.bfloat16, scale=0.2), rnd(N, seed=9)
    z = x.float() @ w.float().T + bias
    want = torch.relu(z) ** 2
    assert rel(torch.relu(z), want) > 0.05 and rel(z, want) > 0.05
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    kernels = []
    if M <= o.SKINNY_MAX_TOKENS:
        kernels += [lambda *a, **k: o.gemm_tc_swap(*a, status=status, **k)]
        if o.skinny_ok(x, w):
            kernels.append(o.gemm_skinny)
    else:
        kernels += [lambda *a, **k: o.gemm_tc(*a, status=status, **k), lambda *a, **k: o.gemm_tc2(*a, status=status, **k)]
    for kern in kernels:
        for dt, tol in ((torch.float32, 3e-5), (torch.bfloat16, TOL["bfloat16"])):
            out = torch.full((M, N), 7.0, dtype=dt, device=DEV)
            kern(x, w, out, bias=bias, unary="relu_square")
            assert int(status) == 0 and rel(out, want) < tol
    for after_short in (False, True):
        out = torch.full((M, N), 7.0, device=DEV)
        o.linear(x, w, out, bias=bias, status=status, activation="relu_square", after_short_kernel=after_short)
        assert int(status) == 0 and rel(out, want) < 3e-5
    x32, w32 = x.float(), w.float()      # 32-bit operands: the generic kernel, then the activation as a step of its own
    out = torch.full((M, N), 7.0, device=DEV)
    o.linear(x32, w32, out, bias=bias, activation="relu_square")
    assert rel(out, want) < 3e-5
    with pytest.raises(o.KernelError):
        o.linear(x, w, out, activation="relu_cube")
    with pytest.raises(o.KernelError):
        o.gemm_tc_swap(x[:1], torch.cat([w, w]), out[:1], gated=True, unary="relu_square")


@pytest.mark.parametrize("M,I,K", [(256, 128, 64), (200, 1408, 256), (70, 100, 96), (2048, 5632, 2048)])
def test_gemm_tc2_gated(M, I, K):
    o = ops()
    x, w = rnd(M, K, dtype=torch.bfloat16), rnd(2 * I, K, dtype=torch.bfloat16, scale=0.2)
    gate, up = x.float() @ w[:I].float().T, x.float() @ w[I:].float().T
    out = torch.empty(M, I, dtype=torch.float32, device=DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    o.gemm_tc2(x, w, out, gated=True, status=status)
    assert int(status) == 0 and rel(out, gate / (1 + torch.exp(-gate)) * up) < 3e-5


@pytest.mark.parametrize("M,I,K", [(128, 64, 64), (200, 1408, 256), (70, 100, 96), (2048, 5632, 2048), (700, 300, 136)])
def test_gemm_tc_gated(M, I, K):
    o = ops()
    x, w = rnd(M, K, dtype=torch.bfloat16), rnd(2 * I, K, dtype=torch.bfloat16, scale=0.2)
    gate, up = x.float() @ w[:I].float().T, x.float() @ w[I:].float().T
    out = torch.empty(M, I, dtype=torch.float32, device=DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    o.gemm_tc(x, w, out, gated=True, status=status)
    assert int(status) == 0 and rel(out, gate / (1 + torch.exp(-gate)) * up) < 3e-5


@pytest.mark.parametrize("counts", [[0, 130, 1, 0, 128, 255], [3, 0, 0, 0, 0, 700], [64, 64, 64, 64, 64, 64],
                                    [137, 0, 512, 9] * 15, [136] * 60, [129, 8, 260, 256, 257, 1, 384, 385, 127, 128],
                                    [1000, 0, 0, 513]])
def test_gemm_tc_grouped(counts):
    o = ops()
    G = len(counts)
    I, H = (96, 128) if G < 10 else (320, 520)   # the large case takes 128 x 256 tiles and several tiles per CTA
    R = sum(counts)
    x = rnd(R, H, dtype=torch.bfloat16)
    w_gu, w_down = rnd(G, 2 * I, H, dtype=torch.bfloat16, scale=0.1), rnd(G, H, I, dtype=torch.bfloat16, scale=0.1)
    offsets = torch.tensor([0] + list(torch.tensor(counts).cumsum(0)), dtype=torch.int32, device=DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    act = torch.full((R, I), 9.0, dtype=torch.bfloat16, device=DEV)
    o.gemm_tc(x, w_gu, act, gated=True, group_offsets=offsets, status=status)
    y = torch.empty(R, H, dtype=torch.float32, device=DEV)
    o.gemm_tc(act, w_down, y, group_offsets=offsets, status=status)
    assert int(status) == 0
    r = 0
    for g, c in enumerate(counts):
        if c == 0:
            continue
        gu = x[r:r + c].float() @ w_gu[g].float().T
        want = gu[:, :I] / (1 + torch.exp(-gu[:, :I])) * gu[:, I:]
        assert rel(act[r:r + c], want) < TOL["bfloat16"], g
        assert rel(y[r:r + c], act[r:r + c].float() @ w_down[g].float().T) < 2e-5, g
        r += c


@pytest.mark.parametrize("M,N,K,tnb", [(40, 300, 136, 0), (17, 128, 64, 32), (64, 2048, 5632, 0), (130, 520, 264, 0),
                                       (300, 200, 96, 64), (5, 61, 2048, 0)])
def test_gemm_tc_swap(M, N, K, tnb):
    """Features in the lanes, tokens in the columns: plain, with bias, accumulating, into a strided view."""
    o = ops()
    x, w = rnd(M, K, dtype=torch.bfloat16), rnd(N, K, dtype=torch.bfloat16, scale=0.2)
    bias = rnd(N, seed=5)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    want = x.float() @ w.float().T
    out = torch.full((M, N), 7.0, dtype=torch.bfloat16, device=DEV)
    o.gemm_tc_swap(x, w, out, bias=bias, tokens_per_tile=tnb, status=status)
    assert int(status) == 0
    assert rel(out, want + bias) < TOL["bfloat16"]
    acc = rnd(M, N, seed=3)
    base = acc.clone()
    o.gemm_tc_swap(x, w, acc, accumulate=True, tokens_per_tile=tnb, status=status)
    assert int(status) == 0 and rel(acc, base + want) < 2e-5
    wide = torch.full((M, N + 5), 7.0, device=DEV)
    o.gemm_tc_swap(x, w, wide[:, :N], tokens_per_tile=tnb, status=status)
    assert rel(wide[:, :N], want) < 2e-5 and float(wide[:, N:].min()) == 7.0


@pytest.mark.parametrize("M,N,K,splits", [(64, 2048, 5632, 8), (40, 300, 136, 3), (17, 128, 64, 1), (5, 61, 2048, 4)])
def test_gemm_tc_swap_runs_of_k(M, N, K, splits):
    """K cut into runs taken by separate CTAs, partial sums added in run order: bias, accumulation, a strided view;
    the same bits every time."""
    o = ops()
    x, w = rnd(M, K, dtype=torch.bfloat16), rnd(N, K, dtype=torch.bfloat16, scale=0.2)
    bias = rnd(N, seed=5)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    want = x.float() @ w.float().T
    out = torch.full((M, N), 7.0, dtype=torch.bfloat16, device=DEV)
    o.gemm_tc_swap(x, w, out, bias=bias, k_splits=splits, status=status)
    assert int(status) == 0 and rel(out, want + bias) < TOL["bfloat16"]
    acc = rnd(M, N, seed=3)
    base = acc.clone()
    o.gemm_tc_swap(x, w, acc, accumulate=True, k_splits=splits, status=status)
    assert int(status) == 0 and rel(acc, base + want) < 2e-5
    wide = torch.full((M, N + 5), 7.0, device=DEV)
    o.gemm_tc_swap(x, w, wide[:, :N], k_splits=splits, status=status)
    first = wide.clone()
    assert rel(wide[:, :N], want) < 2e-5 and float(wide[:, N:].min()) == 7.0
    for _ in range(3):
        o.gemm_tc_swap(x, w, wide[:, :N], k_splits=splits, status=status)
        assert torch.equal(wide, first)
    if splits > 1:
        with pytest.raises(o.KernelError):   # more runs than there are k-blocks
            o.gemm_tc_swap(x, w, out, k_splits=K // 64 + 2, status=status)


@pytest.mark.parametrize("M,I,K", [(48, 100, 96), (64, 5632, 2048), (33, 1408, 256), (200, 300, 136)])
def test_gemm_tc_swap_gated(M, I, K):
    o = ops()
    x, w = rnd(M, K, dtype=torch.bfloat16), rnd(2 * I, K, dtype=torch.bfloat16, scale=0.2)
    gate, up = x.float() @ w[:I].float().T, x.float() @ w[I:].float().T
    out = torch.empty(M, I, dtype=torch.float32, device=DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    o.gemm_tc_swap(x, w, out, gated=True, status=status)
    assert int(status) == 0 and rel(out, gate / (1 + torch.exp(-gate)) * up) < 3e-5


@pytest.mark.parametrize("counts", [[0, 130, 1, 0, 128, 255], [3, 0, 0, 0, 0, 700], [16, 17, 15, 64, 129, 1],
                                    [137, 0, 512, 9] * 15])
def test_gemm_tc_swap_grouped(counts):
    o = ops()
    G = len(counts)
    I, H = (96, 128) if G < 10 else (320, 520)
    R = sum(counts)
    x = rnd(R, H, dtype=torch.bfloat16)
    w_gu, w_down = rnd(G, 2 * I, H, dtype=torch.bfloat16, scale=0.1), rnd(G, H, I, dtype=torch.bfloat16, scale=0.1)
    offsets = torch.tensor([0] + list(torch.tensor(counts).cumsum(0)), dtype=torch.int32, device=DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    act = torch.full((R, I), 9.0, dtype=torch.bfloat16, device=DEV)
    o.gemm_tc_swap(x, w_gu, act, gated=True, group_offsets=offsets, status=status)
    y = torch.empty(R, H, dtype=torch.float32, device=DEV)
    o.gemm_tc_swap(act, w_down, y, group_offsets=offsets, status=status)
    assert int(status) == 0
    r = 0
    for g, c in enumerate(counts):
        if c == 0:
            continue
        gu = x[r:r + c].float() @ w_gu[g].float().T
        want = gu[:, :I] / (1 + torch.exp(-gu[:, :I])) * gu[:, I:]
        assert rel(act[r:r + c], want) < TOL["bfloat16"], g
        assert rel(y[r:r + c], act[r:r + c].float() @ w_down[g].float().T) < 2e-5, g
        r += c


def test_gather_rows():
    o = ops()
    x = rnd(9, 72, dtype=torch.bfloat16)
    rows = torch.tensor([8, 0, 0, 3, 5], dtype=torch.int32, device=DEV)
    out = torch.empty(5, 72, dtype=torch.bfloat16, device=DEV)
    o.gather_rows(x, rows, out)
    assert torch.equal(out, x[rows.long()])
    xf = rnd(9, 7)
    outf = torch.empty(5, 7, device=DEV)
    o.gather_rows(xf, rows, outf)
    assert torch.equal(outf, xf[rows.long()])


@pytest.mark.parametrize("case", ATT_CASES + [(4, 4, 80, 16, 33, [200, 70]), (2, 2, 16, 4, 0, [129])])
def test_prefill_attention_tiles(case):
    """Prompt portions (whole prompts and continuations after a cached prefix) through
    the tiled tensor-core kernel, against the plain per-query statement."""
    o = ops()
    nh, nkv, d, ps, window, lens = case
    dt = torch.bfloat16
    kp, vp, table, ks, vs = build_cache(dt, lens, nkv, d, ps, n_pages=sum(-(-L // ps) for L in lens) + 3, seed=2)
    starts = [0 if i % 2 == 0 else min(L - 1, max(1, L // 3)) for i, L in enumerate(lens)]
    toks, tiles, flat = [], [], 0
    for s, (L, st) in enumerate(zip(lens, starts)):
        n = L - st
        for i in range(0, n, 64):
            tiles.append((flat + i, min(64, n - i), s, st + i))
        toks += [(s, p) for p in range(st, L)]
        flat += n
    T = len(toks)
    q = rnd(T, nh * d + 2 * nkv * d, dtype=dt, seed=T)
    tiles_t = torch.tensor(tiles, dtype=torch.int32, device=DEV)
    seq_slot = torch.tensor([s + 1 for s in range(len(lens))], dtype=torch.int32, device=DEV)
    out = torch.zeros(T, nh * d, dtype=dt, device=DEV)
    scale = 1 / math.sqrt(d)
    o.prefill_attention(q, kp, vp, table, ps, tiles_t, seq_slot, out, nh, nkv, d, window, scale)
    assert torch.isfinite(out.float()).all()
    step = max(1, T // 40)  # a spread of tokens, plus tile edges
    check = sorted(set(list(range(0, T, step)) + [t for t in (0, 1, 63, 64, 65, 127, 128, T - 1) if t < T]))
    for i in check:
        s, pos = toks[i]
        want = plain_attention(q[i, : nh * d].float().cpu().reshape(nh, d), ks[s], vs[s], pos, window, scale)
        assert rel(out[i].float().cpu().reshape(nh, d), want) < 1.5e-2, (i, s, pos)


def mma_attention(kernel, q, kp, vp, table, page, portions, nh, nkv, window=0, scale=1.0, **options):
    """The mma.sync prompt attention ("prefill") or that of the general form ("general", options as it takes them) over
    portions of (slot, first position, tokens); q [tokens, nh * d] bfloat16."""
    o = ops()
    as_int = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    d, dv = kp.shape[-1], vp.shape[-1]
    out = torch.full((q.shape[0], nh * dv), float("nan"), dtype=torch.bfloat16, device=DEV)
    slots = as_int([s for s, _, _ in portions])
    if kernel == "prefill":
        tiles, flat = [], 0
        for b, (_, start, n) in enumerate(portions):
            tiles += [(flat + i, min(64, n - i), b, start + i) for i in range(0, n, 64)]
            flat += n
        return o.prefill_attention(q, kp, vp, table, page, as_int(tiles), slots, out, nh, nkv, d, window, scale, **options)
    positions = as_int([p for _, start, n in portions for p in range(start, start + n)])
    seq = as_int([b for b, (_, _, n) in enumerate(portions) for _ in range(n)])
    items = torch.from_numpy(o.general_attention_items([n for _, _, n in portions], nh, nkv)).to(DEV)
    return o.general_attention(q, q.stride(0), d, kp, vp, d, dv, table, page, positions, seq, slots, items, out, nh * dv, dv,
                               nh, nkv, d, dv, window, scale, **options)


@pytest.mark.parametrize("kernel", ["prefill", "general"])
def test_prompt_attention_on_mma_keeps_32_bit_scores_and_weights(kernel):
    """A cap far above the scores leaves them as they are (a tanh whose error is absolute would not: 3e-7 of 1e7), and a weight
    below the smallest normal number still counts (it is rounded to 16 bits: 2^-130 to three bits)."""
    lens, nh, nkv, d, page = [70], 2, 1, 64, 32
    kp, vp, table, ks, vs = build_cache(torch.bfloat16, lens, nkv, d, page, n_pages=4)
    q = rnd(70, nh * d, dtype=torch.bfloat16)
    run = lambda q, kp, vp, **kw: mma_attention(kernel, q, kp, vp, table, page, [(1, 0, q.shape[0])], nh, nkv, **kw)
    out = run(q, kp, vp, scale=d ** -0.5, softcap=1e7)
    for t in range(70):
        want = plain_attention(q[t].float().cpu().view(nh, d), ks[0], vs[0], t, 0, d ** -0.5)
        assert rel(out[t].float().cpu().view(nh, d), want) < 1.5e-2, t
    q, kp, vp = torch.zeros(2, nh * d, dtype=torch.bfloat16, device=DEV), torch.zeros_like(kp), torch.zeros_like(vp)
    first = int(table[1, 0])
    q[:, ::d], kp[first, 0, 1, 0], vp[first, 0, 1] = 1.0, -90.0, 1e38
    got, want = run(q, kp, vp).double(), math.exp(-90.0) * float(vp[first, 0, 1, 0])
    assert bool((got[0] == 0).all()) and bool(((got[1] - want).abs() < want / 8).all())


EDGES = [     # kernel, head widths of keys and values, page, options
    ("prefill", 64, 64, 32, {}), ("prefill", 48, 48, 96, dict(window=33)), ("prefill", 128, 128, 64, dict(window=64)),
    ("prefill", 64, 64, 4, dict(window=97)), ("general", 64, 64, 64, {}), ("general", 64, 128, 96, dict(window=65)),
    ("general", 48, 80, 32, dict(window=64, keep_first=4)), ("general", 64, 64, 64, dict(window=32, keep_first=70)),
    ("general", 192, 128, 32, dict(window=31, keep_first=33)), ("general", 64, 64, 64, dict(chunk=64)),
    ("general", 80, 48, 20, dict(chunk=100)), ("general", 128, 128, 128, dict(window=128, softcap=5.0)),
]


@pytest.mark.parametrize("kernel,d,dv,page,options", EDGES)
def test_every_query_sees_its_keys_and_no_other(kernel, d, dv, page, options):
    """Queries of zeros weigh all keys that they see alike, and key j's value is the unit vector j mod width: the result counts the
    keys seen, one by one.  Portions that begin and end at and beside the edges of blocks of 32 and 64 keys, windows, kept first
    positions, chunks and pages; and, one token a request, keys cut into runs."""
    o = ops()
    nh, nkv = 4, 2
    portions = [(1, 0, 200), (2, 31, 34), (3, 64, 65), (4, 127, 1), (5, 189, 4), (6, 95, 97)]
    lens = [a + n for _, a, n in portions]
    kp, _, table, _, _ = build_cache(torch.bfloat16, lens, nkv, d, page, n_pages=sum(-(-L // page) for L in lens) + 2)
    # (rows of no request and positions behind a request's last hold what must not be seen)
    vp = torch.full((kp.shape[0], nkv, page, dv), 1e4, dtype=torch.bfloat16, device=DEV)
    for slot, L in enumerate(lens, 1):
        for j in range(L):
            vp[int(table[slot, j // page]), :, j % page] = torch.nn.functional.one_hot(torch.tensor(j % dv), dv).to(DEV)
    window, keep, chunk = (options.get(x) or 0 for x in ("window", "keep_first", "chunk"))

    def seen(pos):
        return [j for j in range(pos + 1) if (not window or j > pos - window or j < keep) and (not chunk or j // chunk == pos // chunk)]

    def check(out, tokens):
        for row, pos in zip(out.double().cpu().view(len(tokens), nh, dv), tokens):
            keys = seen(pos)
            want = torch.bincount(torch.tensor(keys) % dv, minlength=dv).double() / len(keys)
            assert ((row - want).abs() <= 2.0 ** -8 * want).all(), pos

    tokens = [p for _, a, n in portions for p in range(a, a + n)]
    q = torch.zeros(len(tokens), nh * d, dtype=torch.bfloat16, device=DEV)
    check(mma_attention(kernel, q, kp, vp, table, page, portions, nh, nkv, **options), tokens)
    if kernel == "general":
        as_int = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
        last, n = [L - 1 for L in lens], len(lens)
        for splits in (1, 3):
            out = torch.empty(n, nh * dv, dtype=torch.bfloat16, device=DEV)
            part_o, part_ml = torch.empty(n, nh, splits, dv, device=DEV), torch.empty(n, nh, splits, 2, device=DEV)
            o.general_attention(q[:n], q.stride(0), d, kp, vp, d, dv, table, page, as_int(last), as_int(list(range(n))),
                                as_int(list(range(1, n + 1))), None, out, nh * dv, dv, nh, nkv, d, dv, scale=1.0, n_splits=splits,
                                part_o=part_o, part_ml=part_ml, **dict(dict(window=0), **options))
            check(out, last)


TC_ATT_CASES = [
    # nh, nkv, d, page, window, lengths
    (16, 16, 128, 64, 0, [300, 64, 65]),
    (28, 4, 128, 64, 100, [130, 517]),
    (6, 2, 64, 128, 0, [700, 129]),
    (3, 1, 64, 64, 300, [900]),
    (2, 2, 128, 192, 129, [400, 2, 128]),
    (4, 2, 128, 64, 0, [2300, 300]),
    (2, 1, 128, 64, 0, [6000]),
    (2, 2, 64, 64, 2048, [4300]),
]


@pytest.mark.parametrize("run_blocks", [-1, 0, 1, 3])
@pytest.mark.parametrize("case", TC_ATT_CASES)
def test_prefill_attention_tcgen05(case, run_blocks):
    """Prompt portions through the tcgen05 kernel (tiles of 256 queries, blocks of 128 keys), whole prompts and
    continuations after a cached prefix, against the plain per-query statement; with the planner's own cut of
    long tiles into runs of key blocks, and with runs of one and of three blocks (every tile with more is then added
    up from partial results by the second kernel).  One far key of the longest request is made to stand out for its
    last query, so that a block that is skipped or masked wrongly shows."""
    o = ops()
    nh, nkv, d, ps, window, lens = case
    dt = torch.bfloat16
    kp, vp, table, ks, vs = build_cache(dt, lens, nkv, d, ps, n_pages=sum(-(-L // ps) for L in lens) + 3, seed=5)
    # stale finite values in the unused places of every page, as pages that are used again hold
    starts = [0 if i % 2 == 0 else min(L - 1, max(1, L // 3)) for i, L in enumerate(lens)]
    toks = []
    for s, (L, st) in enumerate(zip(lens, starts)):
        toks += [(s, p) for p in range(st, L)]
    T = len(toks)
    items, merges, parts = o.prefill_tc_plan([(L - st, st) for L, st in zip(lens, starts)], window, nh, run_blocks=run_blocks)
    if run_blocks == 1:
        assert parts >= max(lens) // 128 and len(merges) >= 1
    if window:
        # pages that the window has left behind are given back before a later portion runs: no page there
        for s, st in enumerate(starts):
            for j in range(max(0, st - window + 1) // ps):
                table[s + 1, j] = -1
    q = rnd(T, nh * d + 2 * nkv * d, dtype=dt, seed=T)
    # the last query of request 0 looks hard at one far key that is still inside its window
    L0 = lens[0]
    far = max(0, L0 - 1 - (window - 2 if window else L0))
    last0 = L0 - starts[0] - 1
    q[last0, :d] = (ks[0][far, 0] * 4).to(dt).to(DEV)
    seq_slot = torch.tensor([s + 1 for s in range(len(lens))], dtype=torch.int32, device=DEV)
    out = torch.zeros(T, nh * d, dtype=dt, device=DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    scale = 1 / math.sqrt(d)
    assert o.prefill_tc_ok(q, out, kp, ps, d)
    part_o = torch.full((max(parts, 1), nh, 256, d), float("nan"), device=DEV)      # what a run does not write is not read
    part_ml = torch.full((max(parts, 1), nh, 256, 2), float("nan"), device=DEV)
    o.prefill_attention_tc(q, kp, vp, table, ps, torch.from_numpy(items).to(DEV), seq_slot, out, nh, nkv, d, window, scale,
                           status=status, merges=torch.from_numpy(merges).to(DEV) if parts else None, part_o=part_o,
                           part_ml=part_ml)
    assert int(status) == 0
    assert torch.isfinite(out.float()).all()
    step = max(1, T // 40)  # a spread of tokens, plus tile edges
    check = sorted(set(list(range(0, T, step)) + [t for t in (0, 1, 63, 64, 127, 128, 129, 255, 256, last0, T - 1) if t < T]))
    for i in check:
        s, pos = toks[i]
        want = plain_attention(q[i, : nh * d].float().cpu().reshape(nh, d), ks[s], vs[s], pos, window, scale)
        assert rel(out[i].float().cpu().reshape(nh, d), want) < 1.5e-2, (i, s, pos)
    # the far key carries (nearly) all the weight of that query's first head
    got = out[last0, :d].float().cpu()
    assert rel(got, vs[0][far, 0]) < 5e-2


def general_attention_in_64_bits(q, kp, vp, table, lens, starts, H, G, share, window, keep, chunk, cap, scale, sinks):
    """[tokens, H, V] of the general forms, from the pages; q [tokens, H, D]."""
    outs, flat = [], 0
    for b, (n, start) in enumerate(zip(lens, starts)):
        L = start + n
        pages = table[b, :-(-L // kp.shape[2])].long().clamp(min=0)
        K, V = (t[pages].transpose(0, 1).flatten(1, 2)[:, :L].double() for t in (kp, vp))
        i, j = torch.arange(start, L, device=DEV)[:, None], torch.arange(L, device=DEV)[None]
        seen = j <= i
        if window:
            seen &= (j > i - window) | (j < keep)
        if chunk:
            seen &= j // chunk == i // chunk
        out = []
        for h in range(H):
            s = q[flat:flat + n, h].double() @ K[h * G // H].T * scale
            s = (cap * torch.tanh(s / cap) if cap else s).masked_fill(~seen, -math.inf)
            if sinks is not None:
                s = torch.cat([s, sinks[h].double().expand(n, 1)], 1)
            out.append(torch.softmax(s, -1)[:, :L] @ V[h * G // H // share])
        outs.append(torch.stack(out, 1))
        flat += n
    return torch.cat(outs)


# heads, key heads, key heads a value head, D, V, window, keep_first, chunk, cap, sinks, query size, (lengths, starts)
TC_GENERAL = [
    (8, 4, 2, 64, 128, 0, 0, None, 30.0, False, 3.0, ([300, 9], [0, 500])),     # scores up to a sixth of the cap: all by the cubic
    (4, 2, 1, 128, 128, 200, 0, None, 5.0, True, 8.0, ([600], [100])),           # scores beyond the cap: tanhf
    (4, 2, 2, 128, 64, 0, 0, None, 40.0, False, 1.0, ([130, 1], [0, 0])),
    (4, 1, 1, 128, 128, 150, 5, None, None, False, 1.0, ([700, 20], [0, 900])),
    (2, 2, 1, 64, 64, 129, 300, None, None, True, 1.0, ([900], [0])),            # kept blocks that the first tile's own range holds
    (2, 1, 1, 64, 128, 130, 128, None, 20.0, False, 2.0, ([513, 64], [300, 0])),
    (3, 3, 1, 192, 128, 0, 0, None, None, True, 1.0, ([700, 40], [0, 300])),
    (2, 2, 1, 136, 64, 300, 0, None, None, False, 1.0, ([400], [600])),
    (2, 2, 1, 192, 64, 256, 7, None, None, False, 1.0, ([1000], [0])),
    (2, 1, 1, 96, 40, 0, 0, 300, None, False, 1.0, ([700], [50])),
]


@pytest.mark.parametrize("run_blocks", [-1, 0, 1, 2])
@pytest.mark.parametrize("case", TC_GENERAL)
def test_prefill_attention_tcgen05_general(case, run_blocks):
    """The general forms on the tcgen05 kernel: capped scores, kept first positions, shared value heads, wide keys, sinks,
    chunks; tiles whole and cut, strided queries, pages behind a window given back.  Against 64 bits: P and the result are
    rounded to bfloat16 (2^-9 each, a row's P weighted), as in the mma.sync kernels' test."""
    o = ops()
    H, G, share, D, V, window, keep, chunk, cap, with_sinks, size, (lens, starts) = case
    ps, T, n = 64, sum(lens), len(lens)
    width = max(-(-(s + l) // ps) for s, l in zip(starts, lens))
    perm = torch.randperm(n * width + 1, generator=torch.Generator().manual_seed(7))[:n * width].view(n, width)
    table = perm.to(torch.int32).to(DEV)
    kp, vp = rnd(n * width + 1, G, ps, D, dtype=torch.bfloat16, seed=1), rnd(n * width + 1, G // share, ps, V, dtype=torch.bfloat16, seed=2)
    rows = rnd(T, H * D + 16, dtype=torch.bfloat16, seed=3, scale=size)
    q = rows[:, :H * D]
    sinks = rnd(H, seed=4) if with_sinks else None
    scale = D ** -0.5
    want = general_attention_in_64_bits(q.reshape(T, H, D), kp, vp, table, lens, starts, H, G, share, window, keep, chunk, cap, scale, sinks)
    if window:      # pages that no query of the step sees: given back
        for b, s in enumerate(starts):
            table[b, -(-keep // ps):max(-(-keep // ps), (s - window + 1) // ps)] = -1
    items, merges, parts = o.prefill_tc_plan(list(zip(lens, starts)), window, H, run_blocks=run_blocks, chunk=chunk, keep_first=keep)
    part_o = torch.full((max(parts, 1), H, 256, o.prefill_value_width(V)), float("nan"), device=DEV)
    part_ml = torch.full((max(parts, 1), H, 256, 2), float("nan"), device=DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    out = torch.full((T, H * V + 8), 7.0, dtype=torch.bfloat16, device=DEV)
    assert o.prefill_tc_general_ok(q, q.stride(0), D, kp, vp, ps, out, out.stride(0), V, D, V, scale, cap)
    o.prefill_attention_tc(q, kp, vp, table, ps, torch.from_numpy(items).to(DEV), torch.arange(n, dtype=torch.int32, device=DEV),
                           out[:, :H * V], H, G, D, window, scale, status=status, merges=torch.from_numpy(merges).to(DEV) if parts else None,
                           part_o=part_o, part_ml=part_ml, value_dim=V, chunk=chunk, sinks=sinks, q_strides=(q.stride(0), D),
                           keep_first=keep, softcap=cap, value_share=share, general=True)
    assert int(status) == 0 and bool((out[:, H * V:] == 7).all())
    got = out[:, :H * V].reshape(T, H, V).double()
    assert rel(got, want) < 4e-3
    err = (got - want).flatten(1).norm(dim=1) / want.flatten(1).norm(dim=1)
    assert float(err.max()) < 1.2e-2


def test_prefill_attention_tcgen05_keys_and_values_side_by_side():
    """Rows that hold all heads' keys and values next to each other, reached by strides, are what pages of their own are."""
    o = ops()
    H, D, V, ps, n_pages, T = 3, 192, 128, 128, 4, 300
    wide = H * (D + V)
    kv = rnd(n_pages * ps, wide, dtype=torch.bfloat16, seed=1)
    kp = kv[:, :H * D].reshape(n_pages, ps, H, D).transpose(1, 2).contiguous()
    vp = kv[:, H * D:].reshape(n_pages, ps, H, V).transpose(1, 2).contiguous()
    q = rnd(T, H * D, dtype=torch.bfloat16, seed=2)
    table = torch.tensor([[2, 0, 3, 1]], dtype=torch.int32, device=DEV)
    items, merges, parts = o.prefill_tc_plan([(T, 150)], None, H, run_blocks=0)
    slot = torch.zeros(1, dtype=torch.int32, device=DEV)
    outs = []
    for k, v, strides in ((kp, vp, None), (kv, kv[:, H * D:], (ps * wide, D, wide, ps * wide, V, wide))):
        out = torch.empty(T, H * V, dtype=torch.bfloat16, device=DEV)
        o.prefill_attention_tc(q, k, v, table, ps, torch.from_numpy(items).to(DEV), slot, out, H, H, D, None, D ** -0.5, value_dim=V,
                               kv_strides=strides, n_pages=n_pages, general=True)
        outs.append(out)
    assert torch.equal(*outs)


# heads, key heads, key heads a value head, D, V, window, keep_first, cap, general: the plain form, capped, kept first keys, shared
# value heads, the latent form's widths
HIDDEN_FORMS = [(4, 2, 1, 128, 128, 150, 0, None, False), (4, 2, 1, 128, 128, 150, 0, 20.0, True), (2, 1, 1, 64, 128, 150, 70, None, True),
                (4, 2, 2, 64, 128, 0, 0, 30.0, True), (2, 2, 1, 192, 128, 0, 0, None, True)]


def poisoned(t, mask):
    """A copy of ``t`` whose elements at ``mask`` are no number, infinite and minus infinite in turn."""
    bad = torch.tensor([math.nan, math.inf, -math.inf], dtype=t.dtype, device=t.device)
    at = torch.arange(t.numel(), device=t.device).view(t.shape) % 3
    return torch.where(mask, bad[at], t)


@pytest.mark.parametrize("run_blocks", [0, 1])
@pytest.mark.parametrize("form", HIDDEN_FORMS)
def test_prefill_attention_tcgen05_leaves_out_what_nobody_sees(form, run_blocks):
    """Infinite values and no numbers behind a request's last position, before its window, in pages given back and in page 0, which is
    nobody's here: the bits are those over zeros.  Ends in the first and in the second half of a key block, tiles of one and two
    sub-tiles, portions that begin inside a block."""
    o = ops()
    H, G, share, D, V, window, keep, cap, general = form
    ps, lens, starts = 64, [5, 130, 300, 64, 257], [60, 0, 333, 500, 127]
    T, n, width = sum(lens), len(lens), 11
    n_pages = n * width + 1
    table = (1 + torch.arange(n * width).view(n, width)).to(torch.int32).to(DEV)
    pos = torch.arange(width * ps, device=DEV)
    hidden = torch.ones(n_pages, ps, dtype=torch.bool, device=DEV)
    for b, (L, s) in enumerate(zip(lens, starts)):
        lo = max(0, s - window + 1) if window else 0
        seen = (pos < s + L) & ((pos >= lo) | (pos < keep))
        hidden[table[b].long()] = ~seen.view(width, ps)
        gone = ~seen.view(width, ps).any(1)
        table[b, gone] = -1
    mask = hidden[:, None, :, None]
    kp, vp = rnd(n_pages, G, ps, D, dtype=torch.bfloat16, seed=1), rnd(n_pages, G // share, ps, V, dtype=torch.bfloat16, seed=2)
    q = rnd(T, H * D, dtype=torch.bfloat16, seed=3)
    items, merges, parts = o.prefill_tc_plan(list(zip(lens, starts)), window, H, run_blocks=run_blocks, keep_first=keep)
    outs = []
    for fill in (lambda t: t.masked_fill(mask, 0), lambda t: poisoned(t, mask)):
        part_o = torch.full((max(parts, 1), H, 256, o.prefill_value_width(V)), float("nan"), device=DEV)
        part_ml = torch.full((max(parts, 1), H, 256, 2), float("nan"), device=DEV)
        status, out = torch.zeros(1, dtype=torch.int32, device=DEV), torch.empty(T, H * V, dtype=torch.bfloat16, device=DEV)
        o.prefill_attention_tc(q, fill(kp), fill(vp), table, ps, torch.from_numpy(items).to(DEV), torch.arange(n, dtype=torch.int32, device=DEV),
                               out, H, G, D, window, D ** -0.5, status=status, merges=torch.from_numpy(merges).to(DEV) if parts else None,
                               part_o=part_o, part_ml=part_ml, value_dim=V, keep_first=keep, softcap=cap, value_share=share, general=general)
        assert int(status) == 0
        outs.append(out)
    assert bool(outs[0].isfinite().all()) and torch.equal(*outs)


@pytest.mark.parametrize("D", [64, 128])
def test_prefill_attention_tcgen05_capped_bits_are_the_requests_own(D):
    """A capped request's bits are the same whatever lies behind its last position, before its window, and in the rows of the
    request beside it: scores there are nothing, like its own, a thousand times as large (far beyond where the cap's cubic ends), or
    rise from one key block to the next as its own do not."""
    o = ops()
    H, ps, window, lens, starts = 32, 64, 100, [70, 40], [230, 0]
    n_pages, T = 6, sum(lens)
    kp, vp = rnd(n_pages, H, ps, D, dtype=torch.bfloat16, seed=1), rnd(n_pages, H, ps, D, dtype=torch.bfloat16, seed=2)
    table = torch.tensor([[1, 4, 0, 3, 2], [5, 5, 5, 5, 5]], dtype=torch.int32, device=DEV)
    q = rnd(T, H * D, dtype=torch.bfloat16, seed=3)
    items, _, _ = o.prefill_tc_plan(list(zip(lens, starts)), window, H, run_blocks=0)
    outs = []
    for size in (0, 1, 1000, "rising"):
        k, x = kp.clone(), q.clone()
        if size == "rising":
            x[lens[0]:] = 27 / D ** 0.5 * kp[2, :, 290 - 256].reshape(1, -1)
        else:
            k[2, :, 300 - 256:] *= size
            k[0, :, :(starts[0] - window + 1) - 128] *= size
            x[lens[0]:] *= size
        out = torch.empty(T, H * D, dtype=torch.bfloat16, device=DEV)
        o.prefill_attention_tc(x, k, vp, table, ps, torch.from_numpy(items).to(DEV), torch.arange(2, dtype=torch.int32, device=DEV), out, H, H,
                               D, window, D ** -0.5, softcap=30.0, general=True)
        outs.append(out[:lens[0]])
    assert [torch.equal(outs[0], x) for x in outs[1:]] == [True] * 3


@pytest.mark.parametrize("what", ["raised", "merged", "sink"])
@pytest.mark.parametrize("cap,shift", [(None, 130.0), (40.0, 104.0)])
def test_prefill_attention_tcgen05_small_weights_of_large_values(cap, shift, what):
    """Keys whose weights are 2^-130 of the largest (capped scores: 2^-104, of 2^-115 that they can be) but whose values make up for it
    are in the result: where the row's reference is raised past them, where their run is merged, and under a large sink."""
    o = ops()
    D, ps, T, start = 64, 64, 60, 130
    scale = math.log(2.0) / 8            # the score of (8, 0, ..) and (x, 0, ..) is x powers of two
    if cap:
        half = cap * math.atanh(shift / 2 * math.log(2.0) / cap) / math.log(2.0)
        low, high = -half, half
    else:
        low, high = 0.0, shift
    n_pages, large = 3, 100 if cap is None else 80
    kp, vp = torch.zeros(n_pages, 1, ps, D), torch.full((n_pages, 1, ps, D), 2.0 ** large)
    kp[:, :, :, 0] = low
    sinks = None
    if what == "sink":
        sinks = torch.full((1,), (high if cap is None else shift / 2) * math.log(2.0), device=DEV)
    else:
        kp[2, :, :, 0] = high
        vp[2] = 2.0 ** (large - shift + 5)
    kp, vp = kp.to(DEV, torch.bfloat16), vp.to(DEV, torch.bfloat16)
    q = torch.zeros(T, D, dtype=torch.bfloat16, device=DEV)
    q[:, 0] = 8.0
    table = torch.arange(n_pages, dtype=torch.int32, device=DEV)[None]
    items, merges, parts = o.prefill_tc_plan([(T, start)], None, 1, run_blocks=1 if what == "merged" else 0)
    part_o, part_ml = torch.empty(max(parts, 1), 1, 256, 64, device=DEV), torch.empty(max(parts, 1), 1, 256, 2, device=DEV)
    out = torch.empty(T, D, dtype=torch.bfloat16, device=DEV)
    o.prefill_attention_tc(q, kp, vp, table, ps, torch.from_numpy(items).to(DEV), torch.zeros(1, dtype=torch.int32, device=DEV), out, 1, 1, D, None,
                           scale, merges=torch.from_numpy(merges).to(DEV) if parts else None, part_o=part_o, part_ml=part_ml, sinks=sinks,
                           softcap=cap, general=True)
    want = general_attention_in_64_bits(q.view(T, 1, D), kp, vp, table, [T], [start], 1, 1, 1, 0, 0, None, cap, scale, sinks)
    # the cap's exponent of up to 58 and the scale's of 130 are held to 2^-18: their sum in the weight to 2^-16, the result to 2^-9
    assert float(((out.view(T, 1, D).double() - want).abs() / want).max()) < 2 ** -8


@pytest.mark.parametrize("run_blocks", [0, 1])
@pytest.mark.parametrize("form", [*HIDDEN_FORMS, "turned and gated"])
def test_prefill_attention_tcgen05_values_reach_only_who_sees_them(form, run_blocks):
    """Values that are no numbers or infinite at positions that some of a tile's queries see: what sees one has none in that element;
    what does not has its result, made again in another order of sums (32-bit sums of weights that bfloat16 holds: their rounding, and
    the result's to bfloat16, which may fall to either side); elements beside them keep their bits."""
    o = ops()
    more = form == "turned and gated"
    H, G, share, D, V, window, keep, cap, general = HIDDEN_FORMS[0] if more else form
    ps, T, start = 64, 500, 100
    n_pages = -(-(start + T) // ps)
    table = torch.randperm(n_pages, generator=torch.Generator().manual_seed(3)).to(torch.int32).to(DEV)[None]
    kp, vp = rnd(n_pages, G, ps, D, dtype=torch.bfloat16, seed=1), rnd(n_pages, G // share, ps, V, dtype=torch.bfloat16, seed=2)
    bad, heads = vp.clone(), G // share
    places = [(30, 1, math.inf), (170, 3, math.nan), (270, 5, -math.inf), (271, 5, math.inf), (599, V - 1, math.nan)]
    for p, col, x in places:
        bad[int(table[0, p // ps]), heads - 1, p % ps, col] = x
    q = rnd(T, H * D, dtype=torch.bfloat16, seed=3)
    angle = rnd(T, V // 2, seed=5)
    turn = torch.stack([angle.cos(), angle.sin()], -1).reshape(T, V).contiguous() if more else None
    gate = rnd(T, H * V, dtype=torch.bfloat16, seed=6) if more else None
    items, merges, parts = o.prefill_tc_plan([(T, start)], window, H, run_blocks=run_blocks, keep_first=keep)
    outs = []
    for v in (vp, bad):
        part_o = torch.full((max(parts, 1), H, 256, o.prefill_value_width(V)), float("nan"), device=DEV)
        part_ml = torch.full((max(parts, 1), H, 256, 2), float("nan"), device=DEV)
        status, out = torch.zeros(1, dtype=torch.int32, device=DEV), torch.empty(T, H * V, dtype=torch.bfloat16, device=DEV)
        o.prefill_attention_tc(q, kp, v, table, ps, torch.from_numpy(items).to(DEV), torch.zeros(1, dtype=torch.int32, device=DEV), out, H, G, D,
                               window, D ** -0.5, status=status, merges=torch.from_numpy(merges).to(DEV) if parts else None, part_o=part_o,
                               part_ml=part_ml, value_dim=V, keep_first=keep, softcap=cap, value_share=share, general=general, turn=turn,
                               gate=gate)
        assert int(status) == 0
        outs.append(out.view(T, heads, H // heads, V).float())
    clean, got = outs
    pos = torch.arange(start, start + T, device=DEV)
    touched = torch.zeros(T, heads, V, dtype=torch.bool, device=DEV)
    cols = set()
    for p, col, x in places:
        sees = (p <= pos) & ((p > pos - (window or 1 << 30)) | (p < keep))
        for c in ({col, col ^ 1} if more else {col}):         # (a turned pair: both)
            touched[:, heads - 1, c] |= sees
            cols.add(c)
    touched = touched[:, :, None].expand_as(got)
    assert bool(clean.isfinite().all()) and torch.equal(~got.isfinite(), touched)
    same = torch.ones(heads, 1, V, dtype=torch.bool, device=DEV)
    same[heads - 1, :, sorted(cols)] = False
    assert bool((got == clean)[same.expand_as(got)].all())
    # a weight's rounding to bfloat16 may fall to the other side where its score's sum differs in the last bit (2^-8 of the weight,
    # which is at most 1), and so may the result's (2^-8 of it): seldom
    off, size = (got - clean)[~touched], clean[~touched]
    assert float((off.abs() - 2 ** -8 * size.abs()).max()) <= 2 ** -8 * float(vp.float().abs().max()) and float(off.norm() / size.norm()) < 1e-3


def test_prefill_attention_tcgen05_refuses_other_sizes():
    o = ops()
    q = rnd(4, 3 * 136, dtype=torch.bfloat16)
    kp = torch.zeros(2, 1, 64, 136, dtype=torch.bfloat16, device=DEV)
    out = torch.zeros(4, 136, dtype=torch.bfloat16, device=DEV)
    assert not o.prefill_tc_ok(q, out, kp, 64, 136)
    tiles = torch.tensor([[0, 4, 0, 0, 0, 1, -1, 0]], dtype=torch.int32, device=DEV)
    table = torch.zeros(1, 2, dtype=torch.int32, device=DEV)
    slots = torch.zeros(1, dtype=torch.int32, device=DEV)
    with pytest.raises(o.KernelError):
        o.prefill_attention_tc(q, kp, kp, table, 64, tiles, slots, out, 1, 1, 136, 0, 1.0)
    for bad in (dict(softcap=50.0), dict(softcap=-1.0), dict(softcap=30.0, scale=1e-6), dict(value_share=2), dict(keep_first=-1)):
        with pytest.raises(o.KernelError):
            o.prefill_attention_tc(q, kp, kp, table, 64, tiles, slots, out[:, :128], 1, 1, 128, 10, **dict(dict(scale=1.0, general=True), **bad))
    with pytest.raises(o.KernelError):       # the plain kernel has none of the general forms
        o.prefill_attention_tc(q, kp, kp, table, 64, tiles, slots, out[:, :128], 1, 1, 128, 10, 1.0, keep_first=3)


def test_gemm_skinny_transposed_store_and_linear_picks_it_for_narrow_outputs():
    o = ops()
    T, N, K = 300, 61, 256
    x, w = rnd(T, K, dtype=torch.bfloat16), rnd(N, K, dtype=torch.bfloat16, scale=0.1)
    want = x.float() @ w.float().T
    out = torch.full((T, N), 7.0, device=DEV)
    o.gemm_skinny(w, x, out, transposed_out=True)   # roles swapped: w is the few "tokens", x the streamed matrix
    assert rel(out, want) < 2e-5
    wide = torch.full((T, N + 3), 7.0, device=DEV)   # a view with a row pitch of its own
    o.linear(x, w, wide[:, :N])
    assert rel(wide[:, :N], want) < 2e-5 and float(wide[:, N:].min()) == 7.0


# ------------------------------------------------------------------ random weights
@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("shape,mean,std", [((7,), 0.0, 0.02), ((33, 129), 1.0, 0.02), ((5, 64, 48), 0.0, 1.0),
                                            ((1408, 2048), 0.0, 0.02)])
def test_random_weights_are_the_same_bits_on_the_device_and_on_the_cpu(dtype, shape, mean, std):
    """The device draw against the host's statement of the same rule, bit for bit (odd lengths end inside a pair;
    the last shape is one expert matrix at the real width, its checksum compared as well)."""
    from ferrox_b200.weights import random_init as ri

    key = ri.tensor_key(11, f"t{shape}")
    dev = ri.normal(key, shape, DT[dtype], mean, std, device=DEV).cpu()
    cpu = ri.normal(key, shape, DT[dtype], mean, std, device="cpu")
    assert dev.dtype == cpu.dtype == DT[dtype] and dev.shape == cpu.shape == shape
    ibits = torch.int32 if dtype == "float32" else torch.int16
    assert torch.equal(dev.view(ibits), cpu.view(ibits))
    assert int(dev.view(ibits).to(torch.int64).sum()) == int(cpu.view(ibits).to(torch.int64).sum())


def test_a_model_drawn_on_the_device_is_the_model_of_the_folder(tmp_path):
    """Engine.from_random(on_device=True) and a folder written on the CPU for the same configuration and seed hold
    the same weights: their logits are equal bit for bit."""
    from ferrox_b200 import Engine, StepEntry, write_random_model
    from tiny_configs import TINY_B

    folder = write_random_model(str(tmp_path / "m"), TINY_B, seed=5, norm_init="around_one")
    toks = [(i * 37 + 11) % TINY_B["vocab_size"] for i in range(41)]
    outs = []
    for make in (lambda: Engine.from_folder(folder, dtype="float32", page_size=16, n_pages=8, max_slots=2),
                 lambda: Engine.from_random(TINY_B, seed=5, norm_init="around_one", dtype="float32", on_device=True,
                                            page_size=16, n_pages=8, max_slots=2)):
        eng = make()
        slot = eng.open_request()
        outs.append(eng.step([StepEntry(slot, toks, want=list(range(len(toks))))]).cpu())
    assert torch.equal(outs[0], outs[1])


# ------------------------------------------------------------------ the rotary kernel's other pairing rule
@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("nh,nkv,d,rot", [(4, 2, 16, 16), (3, 1, 48, 20), (2, 2, 128, 128)])
def test_rope_adjacent_pairs_with_a_frequency_table(dtype, nh, nkv, d, rot):
    """Pairs (2i, 2i+1) rotated by pos * inv_freq[i] for an arbitrary table (the reference's interleaved form with
    per-band factors, crates/ferrox-core/src/attention.rs:340-352, 319-337); the rest of the head passes through;
    the keys reach their pages as rotated."""
    o, dt = ops(), DT[dtype]
    ps, T = 8, 5
    width = nh * d + 2 * nkv * d
    qkv = rnd(T, width, dtype=dt)
    before = qkv.clone()
    positions = torch.tensor([0, 1, 2, 40, 41], dtype=torch.int32, device=DEV)
    token_seq = torch.tensor([0, 0, 0, 1, 1], dtype=torch.int32, device=DEV)
    seq_slot = torch.tensor([1, 0], dtype=torch.int32, device=DEV)
    table = torch.full((2, 8), -1, dtype=torch.int32)
    table[1, 0], table[0, 5] = 2, 0
    table = table.to(DEV)
    kp = torch.zeros(3, nkv, ps, d, dtype=dt, device=DEV)
    vp = torch.zeros_like(kp)
    inv_freq = (torch.rand(rot // 2, generator=torch.Generator().manual_seed(rot)) + 0.01).to(DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    o.rope_kv_write(qkv, positions, token_seq, seq_slot, inv_freq, rot, kp, vp, table, ps, nh, nkv, d, True, status,
                    pairing=o.PAIR_ADJACENT)
    assert int(status) == 0
    x = before.float().cpu()
    ang = positions.cpu().float()[:, None] * inv_freq.cpu()[None, :]
    cos, sin = torch.cos(ang), torch.sin(ang)
    tol = 2e-6 if dtype == "float32" else 8e-3
    for t in range(T):
        for hh in range(nh + nkv):
            head = x[t, hh * d:(hh + 1) * d]
            want = head.clone()
            a, b = head[0:rot:2], head[1:rot:2]
            want[0:rot:2] = a * cos[t] - b * sin[t]
            want[1:rot:2] = a * sin[t] + b * cos[t]
            assert rel(qkv[t, hh * d:(hh + 1) * d].cpu(), want) < tol
    for t, (pg, off) in {0: (2, 0), 2: (2, 2), 3: (0, 0), 4: (0, 1)}.items():
        assert torch.equal(kp[pg, :, off, :].reshape(-1), qkv[t, nh * d:(nh + nkv) * d])
        assert torch.equal(vp[pg, :, off, :].reshape(-1), before[t, (nh + nkv) * d:])


# ------------------------------------------------------------------ decode attention right after a long write
@pytest.mark.parametrize("page_size,d", [(64, 128), (16, 48)])
def test_decode_attention_waits_for_a_write_of_many_positions(page_size, d):
    """The public entry makes no assumption about the kernel before it: 100 positions of one request are written by
    the rotary kernel and read by the decode attention launched right behind it (more than any early fetch could
    skip), many times over, against the plain attention."""
    o = ops()
    nh, nkv, n_new, L0 = 4, 2, 100, 90
    dt = torch.bfloat16
    scale = 1 / math.sqrt(d)
    n_pages = -(-(L0 + n_new) // page_size) + 1
    table = torch.full((1, n_pages + 2), -1, dtype=torch.int32)
    table[0, :n_pages] = torch.randperm(n_pages, generator=torch.Generator().manual_seed(3)).int()
    table = table.to(DEV)
    seq_slot = torch.zeros(1, dtype=torch.int32, device=DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    for trial in range(5):
        kp = torch.zeros(n_pages, nkv, page_size, d, dtype=dt, device=DEV)
        vp = torch.zeros_like(kp)
        # the old positions, then the new ones in the very launch before the attention
        rows = rnd(L0 + n_new, (nh + 2 * nkv) * d, dtype=dt, seed=trial)
        want_rows = rows.clone()
        pos_all = torch.arange(L0 + n_new, dtype=torch.int32, device=DEV)
        seq_all = torch.zeros(L0 + n_new, dtype=torch.int32, device=DEV)
        o.rope_kv_write(rows[:L0], pos_all[:L0], seq_all[:L0], seq_slot, None, 0, kp, vp, table, page_size, nh, nkv, d,
                        True, status)
        torch.cuda.synchronize()
        out = torch.zeros(n_new, nh * d, dtype=dt, device=DEV)
        n_splits = 3
        pa = torch.empty(n_new, nh, n_splits, d, device=DEV)
        pm = torch.empty(n_new, nh, n_splits, 2, device=DEV)
        o.rope_kv_write(rows[L0:], pos_all[L0:], seq_all[L0:], seq_slot, None, 0, kp, vp, table, page_size, nh, nkv, d,
                        True, status)
        o.decode_attention(rows[L0:], kp, vp, table, page_size, pos_all[L0:], seq_all[L0:], seq_slot, out, nh, nkv, d,
                           0, scale, 0, n_splits, pa, pm)
        torch.cuda.synchronize()
        assert int(status) == 0
        x = want_rows.float().cpu()
        k = x[:, nh * d:(nh + nkv) * d].reshape(-1, nkv, d)
        v = x[:, (nh + nkv) * d:].reshape(-1, nkv, d)
        for i in (0, 1, 37, n_new - 1):
            want = plain_attention(x[L0 + i, :nh * d].reshape(nh, d), k, v, L0 + i, 0, scale)
            assert rel(out[i].float().cpu().reshape(nh, d), want) < 1e-2, (trial, i)


# ------------------------------------------------------------------ decode attention that rotates and stores itself
@pytest.mark.parametrize("nh,nkv,d,ps,window,lens", [
    (16, 16, 128, 64, 0, [300, 64, 65, 1]),
    (28, 4, 128, 64, 100, [130, 517]),
    (40, 2, 64, 128, 0, [150, 260, 129]),       # 20 query heads a kv head: two blocks of heads share a key's tile
    (6, 2, 192, 128, 150, [318, 70]),
    (4, 4, 256, 64, 33, [140, 64]),
])
@pytest.mark.parametrize("rotate", [True, False])
def test_decode_attention_does_the_rotary_kernels_work_itself(nh, nkv, d, ps, window, lens, rotate):
    """One new token a request: the decode attention given the fused rows as projected (store_new) against the
    rotary kernel followed by the decode attention: the same pages bit for bit, the same output within rounding;
    with one and with several key ranges, merged by the kernel and by the merge kernel; and against plain."""
    o, dt = ops(), torch.bfloat16
    assert o.decode_tma_blocks_per_sm(dt, d, ps) > 0
    kp0, vp0, table, ks, vs = build_cache(dt, lens, nkv, d, ps, n_pages=sum(-(-L // ps) for L in lens) + 3, seed=9)
    B = len(lens)
    positions = torch.tensor([L - 1 for L in lens], dtype=torch.int32, device=DEV)     # the new token is each request's last
    token_seq = torch.arange(B, dtype=torch.int32, device=DEV)
    seq_slot = torch.tensor([s + 1 for s in range(B)], dtype=torch.int32, device=DEV)
    qkv0 = rnd(B, (nh + 2 * nkv) * d + 8, dtype=dt, seed=d)[:, :(nh + 2 * nkv) * d]
    inv_freq = (1.0 / torch.pow(torch.tensor(1e4), torch.arange(0, d // 2).float() * 2 / d)).to(DEV) if rotate else None
    cos_sin = None
    if rotate:
        cos_sin = torch.empty(B, d // 2, 2, device=DEV)
        o.rope_table(positions, inv_freq, cos_sin)
    scale = 1 / math.sqrt(d)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    # the two-kernel way
    qkv_a, kp_a, vp_a = qkv0.clone(), kp0.clone(), vp0.clone()
    o.rope_kv_write(qkv_a, positions, token_seq, seq_slot, inv_freq, d if rotate else 0, kp_a, vp_a, table, ps, nh, nkv, d,
                    True, status, cos_sin=cos_sin)
    for n_splits, with_counters in ((1, False), (3, False), (2, True), (5, True)):
        pa, pm = torch.empty(B, nh, n_splits, d, device=DEV), torch.empty(B, nh, n_splits, 2, device=DEV)
        counters = torch.zeros(B * nkv * -(-(nh // nkv) // 16), dtype=torch.int32, device=DEV) if with_counters else None
        want = torch.zeros(B, nh * d, dtype=dt, device=DEV)
        o.decode_attention(qkv_a, kp_a, vp_a, table, ps, positions, token_seq, seq_slot, want, nh, nkv, d, window, scale,
                           0, n_splits, pa, pm, status=status, counters=counters)
        qkv_b, kp_b, vp_b = qkv0.clone(), kp0.clone(), vp0.clone()
        got = torch.zeros_like(want)
        o.decode_attention(qkv_b, kp_b, vp_b, table, ps, positions, token_seq, seq_slot, got, nh, nkv, d, window, scale,
                           0, n_splits, torch.empty_like(pa), torch.empty_like(pm), status=status, counters=counters,
                           store_new=True, write_pages=True, cos_sin=cos_sin, fresh_positions=1)
        assert int(status) == 0
        assert torch.equal(kp_b, kp_a) and torch.equal(vp_b, vp_a), n_splits       # the pages hold the same bits
        assert torch.equal(qkv_b, qkv0)                                            # the rows stay as projected
        assert rel(got, want) < 4e-3, n_splits
        # a layer that reads another layer's cache: nothing is stored, the token's own key still counts
        kp_c, vp_c = kp0.clone(), vp0.clone()
        got_c = torch.zeros_like(want)
        o.decode_attention(qkv0.clone(), kp_c, vp_c, table, ps, positions, token_seq, seq_slot, got_c, nh, nkv, d, window,
                           scale, 0, n_splits, torch.empty_like(pa), torch.empty_like(pm), status=status, counters=counters,
                           store_new=True, write_pages=False, cos_sin=cos_sin)
        assert torch.equal(kp_c, kp0) and torch.equal(got_c, got)
    # and against the plain statement, with the new key and value in their places
    x = qkv_a.float().cpu()
    for s, L in enumerate(lens):
        ks[s][L - 1] = x[s, nh * d:(nh + nkv) * d].reshape(nkv, d)
        vs[s][L - 1] = x[s, (nh + nkv) * d:].reshape(nkv, d)
        ref = plain_attention(x[s, :nh * d].reshape(nh, d), ks[s], vs[s], L - 1, window, scale)
        assert rel(got[s].float().cpu().reshape(nh, d), ref) < 1e-2, s
    # what the kernel cannot do itself is refused, not approximated
    with pytest.raises(o.KernelError):
        o.decode_attention(qkv0.float(), kp0.float(), vp0.float(), table, ps, positions, token_seq, seq_slot,
                           torch.zeros(B, nh * d, device=DEV), nh, nkv, d, window, scale, 0, 1, pa, pm, store_new=True)


# ------------------------------------------------------------------ router product, routing and gather in one launch
@pytest.mark.parametrize("T,E,K,H,extra", [(1, 60, 4, 2048, 1), (8, 60, 4, 2048, 1), (3, 5, 1, 80, 0), (7, 64, 8, 3584, 0),
                                           (2, 131, 6, 520, 1), (5, 8, 3, 128, 1)])
def test_route_fused_is_product_routing_and_gather(T, E, K, H, extra):
    """One cluster does what three kernels do: logits = x . w^T (E router rows and `extra` further rows, 32-bit sums),
    the routing over the first E, and the rows in expert order.  The logits against a 32-bit product, everything else
    equal to route_small run on those very logits, the gathered rows equal to the rows they copy."""
    o = ops()
    x = rnd(T + 1, H + 8, dtype=torch.bfloat16, seed=T)[1:, :H]        # a strided view
    w = rnd(E + extra, H, dtype=torch.bfloat16, scale=0.3, seed=E)
    assert o.route_fused_ok(x, w, E)
    i32 = dict(dtype=torch.int32, device=DEV)
    R = E + extra
    for renorm in (False, True):
        for gather in (True, False):
            logits = torch.full((T, R), float("nan"), device=DEV)
            ids_a, w_a = torch.empty(T, K, **i32), torch.empty(T, K, device=DEV)
            offsets, src, inv = torch.empty(E + 1, **i32), torch.empty(T * K, **i32), torch.empty(T * K, **i32)
            active = torch.empty(min(E, T * K), **i32)
            xp = torch.full((T * K, H), float("nan"), dtype=torch.bfloat16, device=DEV) if gather else None
            o.route_fused(x, w, logits, K, renorm, ids_a, w_a, offsets, src, inv, active, n_experts=E, xp_out=xp)
            assert rel(logits, x.float() @ w.float().T) < 3e-6
            ids_b, w_b = torch.empty(T, K, **i32), torch.empty(T, K, device=DEV)
            off_b, src_b, inv_b = torch.empty(E + 1, **i32), torch.empty(T * K, **i32), torch.empty(T * K, **i32)
            act_b = torch.empty(min(E, T * K), **i32)
            o.route_small(logits, K, renorm, ids_b, w_b, off_b, src_b, inv_b, act_b, n_experts=E)
            assert torch.equal(ids_a, ids_b) and torch.equal(w_a, w_b) and torch.equal(offsets, off_b)
            assert torch.equal(active, act_b)
            flat = ids_a.flatten().tolist()
            assert sorted(inv.tolist()) == list(range(T * K))
            for i, r in enumerate(inv.tolist()):
                assert int(offsets[flat[i]]) <= r < int(offsets[flat[i] + 1]) and int(src[r]) == i // K
            if gather:
                assert torch.equal(xp, x[src.long()])
    # what it does not take is said beforehand
    assert not o.route_fused_ok(rnd(9, H, dtype=torch.bfloat16), w, E) and not o.route_fused_ok(x.float(), w, E)


# ------------------------------------------------------------------ recurrences in chunks
def scan_setup(lens, seed):
    """(token_seq, seq_slot, tiles of 32 tokens) of entries of these lengths."""
    seq, tiles, flat = [], [], 0
    for b, n in enumerate(lens):
        seq += [b] * n
        tiles += [(flat + i, min(32, n - i), b, i) for i in range(0, n, 32)]
        flat += n
    as_int = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    return as_int(seq), as_int([(b + 2) % (len(lens) + 2) for b in range(len(lens))]), as_int(tiles)


def scan_scratch(*shape):
    return torch.full(shape, float("nan"), device=DEV)


# (entries' lengths, heads, key heads, D, V)
SCANS = [([1], 2, 1, 64, 16), ([31, 32, 33], 4, 2, 128, 128), ([100], 3, 3, 20, 36), ([65, 1, 64], 2, 2, 68, 4),
         ([200, 7], 2, 1, 128, 100), ([64, 5, 97], 4, 2, 64, 48)]


@pytest.mark.parametrize("case", SCANS)
@pytest.mark.parametrize("kind", ["delta", "mlstm"])
def test_chunk_scan(case, kind):
    """The chunked recurrences against the loop over the tokens in 64 bits: decays from nothing to one, states that
    are not empty, slots unlike entries; at one shape and seed within 2e-6 of it or 1.5 times as far as the kernels that take the
    tokens one by one (test_chunked_recurrences_are_as_near_to_64_bits_as_token_by_token holds the mean over many to 1); and what
    is no number in a token reaches no token before it and no other request."""
    o = ops()
    lens, H, G, D, V = case
    G = H if kind == "mlstm" else G
    T, (seq, slot, tiles) = sum(lens), scan_setup(lens, 0)
    wide = rnd(T, 2 * G * D + H * V + 4)
    q, k, v = wide[:, :G * D], wide[:, G * D:2 * G * D], wide[:, 2 * G * D:2 * G * D + H * V]
    n_slots = len(lens) + 2
    state = rnd(n_slots, H, V, D, seed=3)
    gen = torch.Generator().manual_seed(T)
    g = torch.sigmoid(torch.randn(T, H, generator=gen) * 3 + 2)
    g[T // 2] = 0.0
    g[T // 3] = 1.0
    beta = torch.rand(T, H, generator=gen)
    g, beta = g.to(DEV), beta.to(DEV)
    if kind == "delta":
        k.div_(k.reshape(T, G, D).norm(dim=-1, keepdim=True).expand(T, G, D).reshape(T, G * D))
    gates, ib, fb, cap = rnd(T, 2 * H, seed=9) * 4, rnd(H, seed=1), rnd(H, seed=2) + 2, 15.0
    copies = o.mlstm_column_blocks(D, V)
    norm0 = rnd(n_slots, H, 1, D, seed=4).expand(n_slots, H, copies, D).contiguous()
    max0 = rnd(n_slots, H, 1, seed=5).expand(n_slots, H, copies).contiguous()

    def run(chunked, q=q, k=k, v=v):
        st, out, nm, mx = state.clone(), torch.empty(T, H * V, device=DEV), norm0.clone(), max0.clone()
        args = (seq, slot, len(lens))
        if kind == "mlstm" and chunked:
            keep, take, floor = (torch.empty(T, H, device=DEV) for _ in range(3))
            before = torch.empty(len(lens), H, D, device=DEV)
            o.mlstm_gates(gates, ib, fb, cap, mx, nm, before, keep, take, floor, *args, H, D)
            o.chunk_scan(q, k, v, keep, st, out, tiles, *args, H, G, D, V, take=take, q_scale=D ** -0.5, scratch=scan_scratch,
                         normalizer=(before, nm, floor))
        elif kind == "mlstm":
            o.mlstm_scan(q, k, v, gates, ib, fb, cap, D ** -0.5, st, nm, mx, out, *args, H, D, V)
        elif chunked:
            o.chunk_scan(q, k, v, g, st, out, tiles, *args, H, G, D, V, beta=beta, scratch=scan_scratch)
        else:
            o.state_scan(q, k, v, g, H, beta, st, out, *args, H, G, D, V)
        return out, st, nm, mx

    got, old = run(True), run(False)
    d = lambda t: t.double().cpu()
    Q, K = (d(x).view(T, G, D).repeat_interleave(H // G, 1) for x in (q, k))
    Vv, gg, bb = d(v).view(T, H, V), d(g), d(beta)
    want, S_want, n_want = torch.zeros(T, H, V, dtype=torch.float64), d(state), d(norm0)
    for b in range(len(lens)):
        s = int(slot[b])
        S, n, m = S_want[s].transpose(1, 2).clone(), d(norm0)[s, :, 0].clone(), d(max0)[s, :, 0].clone()
        for t in [i for i in range(T) if int(seq[i]) == b]:
            if kind == "delta":
                S = S * gg[t][:, None, None]
                u = bb[t][:, None] * (Vv[t] - torch.einsum("hdv,hd->hv", S, K[t]))
                S = S + K[t][:, :, None] * u[:, None]
                want[t] = torch.einsum("hdv,hd->hv", S, Q[t])
            elif kind == "mlstm":
                gi = cap * torch.tanh((d(gates)[t, :H] + d(ib)) / cap)
                gf = torch.nn.functional.logsigmoid(cap * torch.tanh((d(gates)[t, H:] + d(fb)) / cap))
                mn = torch.maximum(gf + m, gi)
                keep, take = torch.exp(gf + m - mn), torch.exp(gi - mn)
                S = keep[:, None, None] * S + take[:, None, None] * K[t][:, :, None] * Vv[t][:, None]
                n, m = keep[:, None] * n + take[:, None] * K[t], mn
                qs = Q[t] * D ** -0.5
                want[t] = torch.einsum("hdv,hd->hv", S, qs) / (torch.maximum((n * qs).sum(-1).abs(), torch.exp(-m)) + 1e-6)[:, None]
        S_want[s] = S.transpose(1, 2)
        n_want[s] = n[:, None]
    want = want.reshape(T, H * V)
    far = lambda a, b: float((d(a) - b).norm() / b.norm())
    assert far(got[0], want) < max(2e-6, 1.5 * far(old[0], want)) and far(got[1], S_want) < max(1e-6, 1.5 * far(old[1], S_want))
    if kind == "mlstm":
        assert far(got[2], n_want) < 2e-6 and float((got[3] - old[3]).abs().max()) < 1e-5
    t = T // 2
    bad = wide.clone()
    bad[t] = float("nan")
    out = run(True, bad[:, :G * D], bad[:, G * D:2 * G * D], bad[:, 2 * G * D:2 * G * D + H * V])[0]
    keep = [i for i in range(T) if i < t or int(seq[i]) != int(seq[t])]
    assert torch.equal(out[keep], got[0][keep]) and bool(out[t].isnan().any())


@pytest.mark.parametrize("gate", [0, 1])
def test_mlstm_gate_that_is_no_number(gate):
    """A head's input or forget gate that is not a number: its read-outs and states are not from that token on, as token by
    token; the tokens before it, the other head and the other request keep theirs."""
    o = ops()
    lens, H, D, V, cap = [70, 40], 2, 64, 32, 15.0
    T, (seq, slot, tiles) = sum(lens), scan_setup(lens, 0)
    q, k, v, gates = rnd(T, H * D, seed=1), rnd(T, H * D, seed=2), rnd(T, H * V, seed=3), rnd(T, 2 * H, seed=4)
    ib, fb, copies = rnd(H, seed=5), rnd(H, seed=6) + 2, o.mlstm_column_blocks(D, V)
    gates[45, gate * H + 1] = float("nan")

    def run(chunked):
        st, out = torch.zeros(4, H, V, D, device=DEV), torch.empty(T, H * V, device=DEV)
        nm, mx = torch.zeros(4, H, copies, D, device=DEV), torch.zeros(4, H, copies, device=DEV)
        if chunked:
            keep, take, floor = (torch.empty(T, H, device=DEV) for _ in range(3))
            before = torch.empty(2, H, D, device=DEV)
            o.mlstm_gates(gates, ib, fb, cap, mx, nm, before, keep, take, floor, seq, slot, 2, H, D)
            o.chunk_scan(q, k, v, keep, st, out, tiles, seq, slot, 2, H, H, D, V, take=take, q_scale=D ** -0.5,
                         scratch=scan_scratch, normalizer=(before, nm, floor))
        else:
            o.mlstm_scan(q, k, v, gates, ib, fb, cap, D ** -0.5, st, nm, mx, out, seq, slot, 2, H, D, V)
        return [t.isnan() for t in (out, st, nm)]

    got, old = run(True), run(False)
    want = torch.zeros(T, H, V, dtype=torch.bool, device=DEV)
    want[45:70, 1] = True
    assert torch.equal(old[0].view(T, H, V), want)
    for a, b in zip(got, old):
        assert torch.equal(a, b)


@pytest.mark.parametrize("lens,H,D,rank", [([1], 2, 64, 64), ([31, 32, 33], 3, 64, 8), ([100, 5], 2, 20, 3), ([65], 2, 128, 96),
                                           ([130, 1, 64], 1, 100, 65)])
@pytest.mark.parametrize("dtype,rate", [("float32", math.exp(-0.5)), ("bfloat16", math.exp(-0.5)), ("float32", 1.0), ("float32", 0.0)])
def test_chunk_scan_general(dtype, rate, lens, H, D, rank):
    """The generalized delta rule in chunks, from its projections, against the loop in 64 bits, with decays over their whole
    range; at one shape and seed within 2e-6 of it or 1.5 times as far as token by token (the next test holds the mean to 1)."""
    o = ops()
    T, (seq, slot, tiles) = sum(lens), scan_setup(lens, 0)
    wide = rnd(T, 4 * H * D + rank + (-rank) % 4)
    r, k, v, a_pre = (wide[:, i * H * D:(i + 1) * H * D] for i in range(4))
    low, w2, w0 = wide[:, 4 * H * D:4 * H * D + rank], rnd(H * D, rank, dtype=DT[dtype], scale=0.3), rnd(H * D, dtype=DT[dtype], scale=2.0)
    w0[::7], w0[1::7] = 30.0, -30.0            # channels that forget as fast as they can, and that never do
    a_bias = rnd(H * D, dtype=DT[dtype], seed=2)
    state = rnd(len(lens) + 2, H, D, D, seed=3)
    st, st_old = state.clone(), state.clone()
    out, old = torch.empty(T, H * D, device=DEV), torch.empty(T, H * D, device=DEV)
    u, au, w = (torch.empty(T, H * D, device=DEV) for _ in range(3))
    o.general_delta_prep(k, a_pre, low, w2, w0, a_bias, rate, u, au, w, H, D)
    o.general_delta_scan(r, k, v, u, au, w, st_old, old, seq, slot, len(lens), H, D)
    o.chunk_scan_general(r, k, v, a_pre, low, w2, w0, a_bias, rate, st, out, tiles, seq, slot, len(lens), H, D, scratch=scan_scratch)
    d = lambda t: t.double().cpu()
    R, K, Vv = (d(x).reshape(T, H, D) for x in (r, k, v))
    U = K / torch.sqrt((K * K).sum(-1, keepdim=True) + 1e-6)
    A = torch.sigmoid(d(a_pre) + d(a_bias)).view(T, H, D) * U
    W = torch.exp(-rate * torch.sigmoid(torch.tanh(d(low)) @ d(w2).T + d(w0))).view(T, H, D)
    want, S_want = torch.zeros(T, H, D, dtype=torch.float64), d(state)
    for b in range(len(lens)):
        S = S_want[int(slot[b])].transpose(1, 2).clone()
        for t in [i for i in range(T) if int(seq[i]) == b]:
            y = torch.einsum("hi,hij->hj", U[t], S)
            S = W[t][:, :, None] * S - A[t][:, :, None] * y[:, None] + K[t][:, :, None] * Vv[t][:, None]
            want[t] = torch.einsum("hij,hi->hj", S, R[t])
        S_want[int(slot[b])] = S.transpose(1, 2)
    far = lambda a, b: float((d(a) - b).norm() / b.norm())
    want = want.reshape(T, H * D)
    assert far(out, want) < max(2e-6, 1.5 * far(old, want)) and far(st, S_want) < max(1e-6, 1.5 * far(st_old, S_want))


@pytest.mark.parametrize("kind,rate", [("delta", 0), ("mlstm", 0), ("general", math.exp(-0.5)), ("general", 1.0)])
def test_chunked_recurrences_are_as_near_to_64_bits_as_token_by_token(kind, rate):
    """The chunked recurrences' error against the loop in 64 bits, beside that of the kernels that take the tokens one by one:
    summed over shapes and seeds, so that chance evens out, it is no larger (5 % for what chance is left).  An mLSTM's state
    stands for S e^m (its read-outs are quotients, and what their nearly vanishing denominators do to an error is chance)."""
    o = ops()
    d = lambda t: t.double()
    far = lambda a, b: float((d(a) - b).norm() / b.norm())
    new, old = [0.0, 0.0], [0.0, 0.0]
    for lens, H, G, D, V in (([1], 2, 1, 64, 16), ([31, 32, 33], 4, 2, 128, 128), ([100], 3, 3, 20, 36), ([65, 1, 64], 2, 2, 68, 4),
                             ([200, 7], 2, 1, 128, 100), ([64, 5, 97], 4, 2, 64, 48), ([600], 2, 2, 128, 128)):
        G, V = (G if kind == "delta" else H), (D if kind == "general" else V)
        T, n, (seq, slot, tiles) = sum(lens), len(lens), scan_setup(lens, 0)
        at, copies = (seq, slot, n), o.mlstm_column_blocks(D, V)
        for seed in range(12 if kind == "mlstm" else 4):
            gen = torch.Generator(device=DEV).manual_seed(seed)
            rand = lambda *shape: torch.randn(*shape, generator=gen, device=DEV)
            q, k, v, state = rand(T, G * D), rand(T, G * D), rand(T, H * V), rand(n + 2, H, V, D)
            outs, states = [torch.empty(T, H * V, device=DEV) for _ in range(2)], [state.clone(), state.clone()]
            if kind == "delta":
                k = torch.nn.functional.normalize(k.view(T, G, D), dim=-1).view(T, -1).contiguous()
                g, beta = torch.sigmoid(rand(T, H) * 3 + 2), torch.sigmoid(rand(T, H))
                o.chunk_scan(q, k, v, g, states[0], outs[0], tiles, *at, H, G, D, V, beta=beta, scratch=scan_scratch)
                o.state_scan(q, k, v, g, H, beta, states[1], outs[1], *at, H, G, D, V)
            elif kind == "mlstm":
                gates, ib, fb, cap = rand(T, 2 * H) * 4, rand(H), rand(H) + 2, 15.0
                n0 = rand(n + 2, H, 1, D).expand(n + 2, H, copies, D).contiguous()
                m0 = rand(n + 2, H, 1).expand(n + 2, H, copies).contiguous()
                norm, top = [n0.clone(), n0.clone()], [m0.clone(), m0.clone()]
                keep, take, floor = (torch.empty(T, H, device=DEV) for _ in range(3))
                was = torch.empty(n, H, D, device=DEV)
                o.mlstm_gates(gates, ib, fb, cap, top[0], norm[0], was, keep, take, floor, *at, H, D)
                o.chunk_scan(q, k, v, keep, states[0], outs[0], tiles, *at, H, H, D, V, take=take, q_scale=D ** -0.5,
                             scratch=scan_scratch, normalizer=(was, norm[0], floor))
                o.mlstm_scan(q, k, v, gates, ib, fb, cap, D ** -0.5, states[1], norm[1], top[1], outs[1], *at, H, D, V)
            else:
                a_pre, low, w2, w0, ab = rand(T, H * D), rand(T, 64), rand(H * D, 64) * 0.3, rand(H * D) * 2, rand(H * D)
                w0[::7], w0[1::7] = 30.0, -30.0
                o.chunk_scan_general(q, k, v, a_pre, low, w2, w0, ab, rate, states[0], outs[0], tiles, *at, H, D, scratch=scan_scratch)
                u, au, w = (torch.empty(T, H * D, device=DEV) for _ in range(3))
                o.general_delta_prep(k, a_pre, low, w2, w0, ab, rate, u, au, w, H, D)
                o.general_delta_scan(q, k, v, u, au, w, states[1], outs[1], *at, H, D)
                U = d(k).view(T, H, D)
                U = U / torch.sqrt((U * U).sum(-1, keepdim=True) + 1e-6)
                A = torch.sigmoid(d(a_pre) + d(ab)).view(T, H, D) * U
                W = torch.exp(-rate * torch.sigmoid(torch.tanh(d(low)) @ d(w2).T + d(w0))).view(T, H, D)
            Q, K = (d(x).view(T, G, D).repeat_interleave(H // G, 1) for x in (q, k))
            X, want, S_want, t = d(v).view(T, H, V), torch.zeros(T, H, V, dtype=torch.float64, device=DEV), d(state), 0
            for b, L in enumerate(lens):
                S = S_want[int(slot[b])].transpose(1, 2)
                m = d(m0)[int(slot[b]), :, 0] if kind == "mlstm" else None
                for t in range(t, t + L):
                    if kind == "delta":
                        S = S * d(g)[t][:, None, None]
                        S = S + K[t][:, :, None] * (d(beta)[t][:, None] * (X[t] - torch.einsum("hdv,hd->hv", S, K[t])))[:, None]
                    elif kind == "general":
                        y = torch.einsum("hi,hij->hj", U[t], S)
                        S = W[t][:, :, None] * S - A[t][:, :, None] * y[:, None] + K[t][:, :, None] * X[t][:, None]
                    else:
                        gi = cap * torch.tanh((d(gates)[t, :H] + d(ib)) / cap)
                        gf = torch.nn.functional.logsigmoid(cap * torch.tanh((d(gates)[t, H:] + d(fb)) / cap))
                        mn = torch.maximum(gf + m, gi)
                        S = torch.exp(gf + m - mn)[:, None, None] * S + torch.exp(gi - mn)[:, None, None] * K[t][:, :, None] * X[t][:, None]
                        m = mn
                    want[t] = torch.einsum("hdv,hd->hv", S, Q[t])
                t += 1
                S_want[int(slot[b])] = S.transpose(1, 2)
                if kind == "mlstm":
                    for i in range(2):
                        states[i] = d(states[i])
                        states[i][int(slot[b])] *= torch.exp(d(top[i])[int(slot[b]), :, 0] - m)[:, None, None]
            for e, i in ((new, 0), (old, 1)):
                e[0] += far(outs[i], want.view(T, -1)) if kind != "mlstm" else 0.0
                e[1] += far(states[i], S_want)
    assert new[0] <= 1.05 * old[0] and new[1] <= 1.05 * old[1], (new, old)


@pytest.mark.parametrize("lens,G,D,H,V", [([128], 1, 128, 1, 4), ([1, 2, 3, 200], 1, 64, 2, 36), ([17, 130, 16, 4], 2, 128, 4, 128),
                                          ([300], 2, 64, 2, 62)])
def test_delta_prep_by_runs(lens, G, D, H, V, monkeypatch):
    """What the delta rule needs before its recurrence, in runs of tokens: entries that begin and end inside a run and
    beside its edges, against the kernel that takes a token a block (the same order of the convolution's sums)."""
    o = ops()
    T, C, n = sum(lens), 2 * G * D + H * V, len(lens)
    seq, slot, _ = scan_setup(lens, 0)
    proj = rnd(T, C + 2 * H + 4 + (-(C + 2 * H)) % 4)
    ba, conv, tail = proj[:, C:], rnd(C, 4, seed=1), rnd(n + 2, 3, C, seed=2)
    a_log, dt = rnd(H, seed=3), rnd(H, seed=4)

    def run(runs):
        monkeypatch.setattr(o, "DELTA_PREP_RUNS_MIN_TOKENS", 1 if runs else 1 << 30)
        got = torch.empty(T, C, device=DEV), torch.empty(T, H, device=DEV), torch.empty(T, H, device=DEV)
        o.delta_prep(proj, conv, 4, tail, ba, a_log, dt, seq, slot, *got, G, D, H, V)
        return got

    for a, b in zip(run(True), run(False)):
        assert rel(a, b) < 1e-6


@pytest.mark.parametrize("hidden", [4, 100, 1028, 2048, 4100, 8192, 8196, 2046])
@pytest.mark.parametrize("n_rows", [1, 3, 300])
def test_layer_norms_with_the_row_in_registers(n_rows, hidden):
    """Layer norm, and layer norm with the residual addition and the next norm, at the edges of a block's pieces (and
    beyond what the vector form takes), in place, with picked rows, 16- and 32-bit operands; against 64 bits."""
    o, eps = ops(), 1e-5
    ln = lambda x, w, b=0.0: (x - x.mean(-1, keepdim=True)) / torch.sqrt(x.var(-1, unbiased=False, keepdim=True) + eps) * w + b
    x, w, b = rnd(n_rows, hidden) * 3 + 1, rnd(hidden, dtype=torch.bfloat16) + 1, rnd(hidden, seed=4)
    rows = torch.arange(n_rows - 1, -1, -1, dtype=torch.int32, device=DEV)
    for dtype, tol in ((torch.float32, 2e-6), (torch.bfloat16, 1e-2)):
        out = torch.empty(n_rows, hidden, dtype=dtype, device=DEV)
        o.layernorm(x, w, eps, out, rows=rows, bias=b)
        assert rel(out.double(), ln(x.double(), w.double(), b.double()).flip(0)) < tol
    same = x.clone()
    o.layernorm(same, w, eps, same)
    assert rel(same.double(), ln(x.double(), w.double())) < 2e-6
    for dtype, tol in ((torch.float32, 2e-6), (torch.bfloat16, 1e-2)):
        h, y1, y2 = rnd(n_rows, hidden, seed=5), rnd(n_rows, hidden, dtype=dtype, seed=6), rnd(n_rows, hidden, seed=7)
        for second in (None, y2):
            z = 0.5 * y1.double() + (0.25 * y2.double() if second is not None else 0.0)
            want = h.double() + ln(z, w.double())
            got, nxt = h.clone(), torch.empty(n_rows, hidden, dtype=dtype, device=DEV)
            o.layernorm_residual(got, y1, w, eps, scale=0.5, y2=second, scale2=0.25, then=(b, eps, nxt))
            assert rel(got.double(), want) < 2e-6 and rel(nxt.double(), ln(want, b.double())) < 2 * tol


@pytest.mark.parametrize("width", [4, 60, 64, 68, 128, 132, 512, 516, 2048])
@pytest.mark.parametrize("gate_dtype,out_dtype", [(torch.float32, torch.float32), (torch.float32, torch.bfloat16),
                                                  (torch.bfloat16, torch.bfloat16)])
def test_gated_group_norm_over_its_forms(width, gate_dtype, out_dtype):
    """Half a warp, a warp or a block a group, one group or four a thread; numbers of groups that leave a block's last places
    empty; weights shared, an element each, in 16 bits and off a 16-byte boundary.  Tolerance: the row's sum and the products
    in 32 bits (1e-5 with the exponential's 1e-6), and the rounding of the result to its type."""
    g = torch.Generator(device="cuda").manual_seed(width)
    for T, groups, shared, wdt, off in ((1, 1, True, torch.float32, 0), (7, 5, False, torch.bfloat16, 0), (33, 3, True, torch.float32, 1)):
        x = torch.randn(T, groups * width, generator=g, device="cuda")
        rows = torch.randn(T, groups * width + 8, generator=g, device="cuda").to(gate_dtype)
        gate = rows[:, 8:]
        w = torch.randn((width if shared else groups * width) + off, generator=g, device="cuda").to(wdt)[off:]
        for act in ("silu", "sigmoid"):
            out = torch.full((T, groups * width), float("nan"), device="cuda", dtype=out_dtype)
            ops().gated_group_norm(x, gate, w, 1e-5, act, out, groups, width)
            xd, gd = x.double().view(T, groups, width), gate.double().view(T, groups, width)
            want = xd / (xd.square().mean(-1, keepdim=True) + 1e-5).sqrt() * w.double().view(1, 1 if shared else groups, width)
            want = (want * torch.sigmoid(gd) * (gd if act == "silu" else 1)).reshape(T, -1)
            tol = 1e-5 + (0 if out_dtype == torch.float32 else 2.0 ** -8)
            assert ((out.double() - want).abs() <= tol * want.abs() + 1e-6).all()


@pytest.mark.parametrize("width", [4, 32, 60])
def test_gated_group_norm_of_narrow_groups_takes_gates_that_hardly_open(width):
    """sigmoid(-88) is below the smallest normal number, and with large weights it still counts (the quotient of the hardware
    alone answers 0 where its divisor passes 2^126)."""
    x, w = torch.ones(3, 2 * width, device="cuda"), torch.full((2 * width,), 1e30, device="cuda")
    gate = torch.full((3, 2 * width), -88.0, device="cuda")
    for act in ("silu", "sigmoid"):
        out = torch.empty(3, 2 * width, device="cuda", dtype=torch.bfloat16)
        ops().gated_group_norm(x, gate, w, 1e-5, act, out, 2, width)
        want = 1e30 / (1.0 + math.exp(88.0)) * (-88.0 if act == "silu" else 1.0)
        assert ((out.double() - want).abs() < 2.0 ** -7 * abs(want)).all()


def test_a_slot_of_every_state_is_zeroed_and_no_other():
    from ferrox_b200.kernels.ops import SlotZeroer

    shapes = [((4, 3), torch.float32), ((4, 64, 64), torch.float32), ((4, 5), torch.bfloat16), ((4, 8, 1031), torch.float32)]
    ts = [torch.ones(s, device="cuda", dtype=d) for s, d in shapes]
    SlotZeroer(ts)(2)
    for t in ts:
        assert (t[2] == 0).all() and (t[[0, 1, 3]] == 1).all()


@pytest.mark.parametrize("kind,D", [("delta", 64), ("delta", 128), ("general", 64), ("general", 128)])
def test_chunk_scans_by_a_list_of_walks(kind, D):
    """Which block walks which entry, from a list (longest first) or found in the tokens' entries: the same bits."""
    o = ops()
    lens, H = [33, 1, 100, 64], 3
    T, (seq, slot, tiles) = sum(lens), scan_setup(lens, 0)
    q, k, v, a_pre = (rnd(T, H * D, seed=i) for i in range(4))
    low, w2, w0, ab = rnd(T, 64, seed=5), rnd(H * D, 64, seed=6) * 0.3, rnd(H * D, seed=7), rnd(H * D, seed=8)
    k = torch.nn.functional.normalize(k.view(T, H, D), dim=-1).view(T, -1).contiguous()
    g, beta = torch.sigmoid(rnd(T, H, seed=9) * 3 + 2), torch.sigmoid(rnd(T, H, seed=10))
    got = []
    for walks in (None, torch.from_numpy(o.chunk_walks(lens)).to(DEV)):
        st, out = rnd(len(lens) + 2, H, D, D, seed=11), torch.empty(T, H * D, device=DEV)
        if kind == "delta":
            o.chunk_scan(q, k, v, g, st, out, tiles, seq, slot, len(lens), H, H, D, D, beta=beta, walks=walks, scratch=scan_scratch)
        else:
            o.chunk_scan_general(q, k, v, a_pre, low, w2, w0, ab, 0.6, st, out, tiles, seq, slot, len(lens), H, D, walks=walks,
                                 scratch=scan_scratch)
        got.append((out, st))
    assert all(torch.equal(a, b) and bool(a.isfinite().all()) for a, b in zip(*got))
