"""Flash-style attention kernel through the C ABI against the CPU oracle and the
fixtures produced by the reference module."""
import contextlib
import os

import numpy as np
import pytest
import torch
import torch.nn.functional as F

from oracle import patched_ops as po
from tests._util import assert_close, cuda_or_skip, h16

pytestmark = pytest.mark.gpu
T = torch.from_numpy


def _ops():
    from basedxl_b200 import _lib, ops

    return _lib, ops


@contextlib.contextmanager
def _plan(keys, groups, split):
    """Forces tokens per key tile, query tiles per work unit and K/V split (0 = the kernel's choice)."""
    _lib, _ = _ops()
    l = _lib.lib()
    _lib.check(l.bxl_debug_force_attn_tiles(groups, keys), l, kernels=0)
    _lib.check(l.bxl_debug_force_attn_split(split), l, kernels=0)
    try:
        yield
        _lib.device_status()
    finally:
        _lib.check(l.bxl_debug_force_attn_split(0), l, kernels=0)
        _lib.check(l.bxl_debug_force_attn_tiles(0, 0), l, kernels=0)


# every tile width, count of groups at work and split, some forced, some chosen
PLANS = [(0, 0, 0), (64, 3, 1), (64, 3, 2), (64, 3, 4), (64, 2, 1), (64, 2, 4), (64, 1, 2), (128, 2, 1), (128, 2, 2), (128, 2, 4), (128, 1, 1), (128, 1, 4)]


@pytest.mark.parametrize(
    "B,heads,Lq,Lslot,nslots",
    [
        (1, 1, 128, 128, 1),
        (2, 2, 128, 256, 1),
        (1, 2, 256, 128, 3),
        (2, 10, 77, 77, 1),       # ragged query and key tiles
        (2, 10, 512, 77, 1),      # cross-attention: 77 text tokens
        (2, 20, 1024, 128, 2),    # 320 query tiles
        (2, 20, 1024, 77, 1),     # the same count for cross-attention: a CTA each
        (1, 3, 200, 72, 4),       # ragged slots
        (2, 10, 512, 512, 8),     # benchmark shape at world size 8: L = 4096
        (2, 20, 256, 256, 4),     # 1280-level blocks, 4 strips
        (2, 10, 4096, 77, 1),     # 640 CTAs where 592 are resident
        (2, 20, 1024, 256, 1),    # whole key tiles only, of either width
        (4, 20, 384, 100, 2),     # three query tiles a head, ragged slots
    ],
)
def test_attention_core_vs_oracle(B, heads, Lq, Lslot, nslots):
    dev = cuda_or_skip()
    _lib, ops = _ops()
    C = heads * 64
    gen = torch.Generator().manual_seed(B + heads + Lq + Lslot + nslots)
    q = h16(torch.randn(B, Lq, C, generator=gen))
    slots = [h16(torch.randn(B, Lslot, 2 * C, generator=gen)) for _ in range(nslots)]
    ref = po._sdpa_heads(q, torch.cat(slots, dim=1), heads)
    y = ops.attention(q.half().to(dev), [s.half().to(dev) for s in slots], heads)
    _lib.device_status()
    assert_close(y, ref, what=f"attention B{B} h{heads} Lq{Lq} Ls{Lslot} n{nslots}")


def test_attention_large_logits_are_stable():
    dev = cuda_or_skip()
    _lib, ops = _ops()
    gen = torch.Generator().manual_seed(1)
    q = h16(6 * torch.randn(1, 128, 64, generator=gen))
    kv = h16(torch.cat([6 * torch.randn(1, 384, 64, generator=gen), torch.randn(1, 384, 64, generator=gen)], dim=2))
    ref = po._sdpa_heads(q, kv, 1)
    y = ops.attention(q.half().to(dev), [kv.half().to(dev)], 1)
    _lib.device_status()
    assert torch.isfinite(y).all()
    assert_close(y, ref, tol=4e-3, what="attention with large logits")


@pytest.mark.parametrize("n", [2, 4])
def test_self_attention_block_golden(golden_dir, n):
    """Whole patched self-attention block (to_q, fused to_kv, slots read in place,
    to_out) assembled from the library's GEMM and attention kernels."""
    dev = cuda_or_skip()
    _lib, ops = _ops()
    g = np.load(os.path.join(golden_dir, "attention_pp.npz"))
    x, xp = T(g["x"]), T(g["x_prev"])
    wq, wkv, wo, bo, heads = T(g["wq"]), T(g["wkv"]), T(g["wo"]), T(g["bo"]), int(g["heads"])
    d = lambda t: t.half().to(dev)
    xs, xps = torch.chunk(x, n, 1), torch.chunk(xp, n, 1)
    kv_prev = [ops.linear(d(t), d(wkv)) for t in xps]
    kv_now = [ops.linear(d(t), d(wkv)) for t in xs]
    for i in range(n):
        q = ops.linear(d(xs[i]), d(wq))
        for tag, slots in (("stale", [kv_now[j] if j == i else kv_prev[j] for j in range(n)]), ("sync", kv_now), ("local", [kv_now[i]] * n)):
            o = ops.attention(q, slots, heads)
            y = ops.linear(o, d(wo), d(bo))
            assert_close(y, T(g[f"n{n}_i{i}_{tag}_y"]), tol=4e-3, what=f"self-attention block {tag}")
        assert_close(kv_now[i], T(g[f"n{n}_i{i}_published"]), what="published kv")
    _lib.device_status()


def test_cross_attention_block_golden(golden_dir):
    dev = cuda_or_skip()
    _lib, ops = _ops()
    g = np.load(os.path.join(golden_dir, "attention_pp.npz"))
    d = lambda t: t.half().to(dev)
    x, ctx = T(g["x"]), T(g["cross_ctx"])
    q = ops.linear(d(x), d(T(g["cross_wq"])))
    kv = ops.linear(d(ctx), d(T(g["cross_wkv"])))
    o = ops.attention(q, [kv], int(g["heads"]))
    y = ops.linear(o, d(T(g["cross_wo"])), d(T(g["cross_bo"])))
    _lib.device_status()
    assert_close(y, T(g["cross_y"]), tol=4e-3, what="cross-attention block")


def test_benchmark_shape_self_attention():
    """10 heads x 64 on 2 x 4096 x 640 tokens; stale K/V = current + N(0, 0.01); world sizes 2/4/8."""
    dev = cuda_or_skip()
    _lib, ops = _ops()
    gen = torch.Generator().manual_seed(0)
    C, heads, L = 640, 10, 4096
    kv = h16(torch.randn(2, L, 2 * C, generator=gen))
    kv_prev = h16(kv + 0.01 * torch.randn(2, L, 2 * C, generator=gen))
    q = h16(torch.randn(2, L, C, generator=gen))
    for n in (2, 4, 8):
        ls = L // n
        for i in sorted({0, n // 2, n - 1}):  # first, middle and last strip: the fresh slot in every position
            slots = [(kv if j == i else kv_prev)[:, j * ls : (j + 1) * ls] for j in range(n)]
            ref = po._sdpa_heads(q[:, i * ls : (i + 1) * ls], torch.cat(slots, dim=1), heads)
            y = ops.attention(q[:, i * ls : (i + 1) * ls].half().to(dev), [s.half().to(dev).contiguous() for s in slots], heads)
            _lib.device_status()
            assert_close(y, ref, what=f"self-attention strip {i} of n={n}")


@pytest.mark.parametrize("keys,groups", [(0, 0), (64, 1), (64, 2), (64, 3), (128, 1), (128, 2)])
@pytest.mark.parametrize("split", [1, 2, 4])
@pytest.mark.parametrize("B,heads,Lq,Lslot,nslots", [(1, 2, 256, 128, 4), (2, 3, 200, 72, 5), (1, 20, 256, 256, 4), (2, 10, 512, 77, 1), (1, 4, 640, 512, 2)])
def test_attention_kv_split_over_a_cluster(B, heads, Lq, Lslot, nslots, split, keys, groups):
    """The K/V range split over 1, 2 or 4 CTAs per query block and merged through distributed
    shared memory gives the same result (ragged tiles, several slots, odd query-tile counts, one to three
    query tiles whose rows the CTAs of the cluster share out)."""
    dev = cuda_or_skip()
    _lib, ops = _ops()
    if split > nslots * -(-Lslot // (keys or 64)):
        pytest.skip("more splits than key/value tiles")
    C = heads * 64
    gen = torch.Generator().manual_seed(B + heads + Lq + Lslot + nslots)
    q = h16(torch.randn(B, Lq, C, generator=gen))
    slots = [h16(torch.randn(B, Lslot, 2 * C, generator=gen) * (1.0 + 2.0 * i)) for i in range(nslots)]  # very different maxima per slot
    ref = po._sdpa_heads(q, torch.cat(slots, dim=1), heads)
    with _plan(keys, groups, split):
        y = ops.attention(q.half().to(dev), [s.half().to(dev) for s in slots], heads)
    assert_close(y, ref, tol=3e-3, what=f"attention split={split} keys={keys} groups={groups}")


def test_a_forced_plan_that_does_not_fit_is_refused():
    dev = cuda_or_skip()
    _lib, ops = _ops()
    q, kv = torch.zeros(1, 300, 64, dtype=torch.float16, device=dev), torch.zeros(1, 100, 128, dtype=torch.float16, device=dev)
    with pytest.raises(_lib.BxlError, match="forced"), _plan(128, 2, 2):
        ops.attention(q, [kv], 1)


def test_self_attention_at_16384_tokens():
    """The 2048 x 2048 image's highest-resolution attention (L = 16384 keys): one head, the
    last of 4 strips (4096 queries), stale K/V in the other three slots."""
    dev = cuda_or_skip()
    _lib, ops = _ops()
    gen = torch.Generator().manual_seed(5)
    C, heads, L, n = 64, 1, 16384, 4
    kv = h16(torch.randn(1, L, 2 * C, generator=gen))
    kv_prev = h16(kv + 0.01 * torch.randn(1, L, 2 * C, generator=gen))
    q = h16(torch.randn(1, L, C, generator=gen))
    ls, i = L // n, n - 1
    slots = [(kv if j == i else kv_prev)[:, j * ls : (j + 1) * ls] for j in range(n)]
    ref = po._sdpa_heads(q[:, i * ls : (i + 1) * ls], torch.cat(slots, dim=1), heads)
    y = ops.attention(q[:, i * ls : (i + 1) * ls].half().to(dev), [s.half().to(dev).contiguous() for s in slots], heads)
    _lib.device_status()
    assert_close(y, ref, what="self-attention L=16384")


@pytest.mark.parametrize("keys,groups,split", PLANS)
@pytest.mark.parametrize("Lq", [1, 128, 129, 257, 385, 770])
@pytest.mark.parametrize("Lslot,nslots", [(1, 3), (63, 2), (64, 4), (65, 2), (127, 2), (129, 4), (200, 8)])
def test_attention_tile_edges(Lq, Lslot, nslots, keys, groups, split):
    """One to three query tiles per unit with the last one ragged, key tiles that end on, before and after a 64- and a
    128-token boundary, more than one ring's worth of them, and clusters that merge the rows of every such unit."""
    dev = cuda_or_skip()
    _lib, ops = _ops()
    if split > nslots * -(-Lslot // (keys or 64)):
        pytest.skip("more splits than key/value tiles")
    B, heads = 2, 3
    C = heads * 64
    gen = torch.Generator().manual_seed(Lq + 1000 * Lslot + nslots)
    q = h16(torch.randn(B, Lq, C, generator=gen))
    slots = [h16(torch.randn(B, Lslot, 2 * C, generator=gen)) for _ in range(nslots)]
    ref = po._sdpa_heads(q, torch.cat(slots, dim=1), heads)
    with _plan(keys, groups, split):
        y = ops.attention(q.half().to(dev), [s.half().to(dev) for s in slots], heads)
    assert_close(y, ref, what=f"attention Lq{Lq} Ls{Lslot} n{nslots} keys{keys} groups{groups} split{split}")


@pytest.mark.parametrize("keys,groups,Lq", [(64, 3, 4 * 384 + 60), (128, 2, 6 * 256 + 60), (64, 2, 6 * 256 + 60)])
def test_attention_walks_many_units(keys, groups, Lq):
    """Two or more units for every CTA, the last unit of every head with one tile: the groups' barriers and the rings of
    keys and queries go round many times, with idle groups in between."""
    dev = cuda_or_skip()
    _lib, ops = _ops()
    B, heads, Lslot = 2, 40, 150
    C = heads * 64
    units = B * heads * -(-Lq // (128 * groups))
    assert units >= 2 * _lib.lib().bxl_sm_count()
    gen = torch.Generator().manual_seed(9)
    q, kv = h16(torch.randn(B, Lq, C, generator=gen)), h16(torch.randn(B, Lslot, 2 * C, generator=gen))
    ref = po._sdpa_heads(q, kv, heads)
    with _plan(keys, groups, 1):
        y = ops.attention(q.half().to(dev), [kv.half().to(dev)], heads)
    assert_close(y, ref, what="attention, many units")


def test_attention_keeps_nan_and_infinite_scores():
    """A NaN in one key makes every row NaN, and a key of infinite score as well (inf - inf); other heads are
    untouched."""
    dev = cuda_or_skip()
    _lib, ops = _ops()
    gen = torch.Generator().manual_seed(10)
    q, kv = torch.randn(1, 200, 128, generator=gen).abs().half(), torch.randn(1, 320, 256, generator=gen).half()
    clean = ops.attention(q.to(dev), [kv.to(dev)], 2)
    for value, token in [(float("nan"), t) for t in range(64, 96)] + [(float("inf"), 70)]:
        bad = kv.clone()
        bad[0, token, 5] = value
        y = ops.attention(q.to(dev), [bad.to(dev)], 2)
        assert torch.isnan(y[..., :64]).all(), (value, token)
        assert torch.equal(y[..., 64:], clean[..., 64:])
    _lib.device_status()


@pytest.mark.parametrize("L", [64, 77, 100, 128, 154, 231])
def test_attention_error_with_peaked_scores(L):
    """The rounding of P to fp16 is relative to the maximum of the first 128 keys (raised only beyond 2^8), so that the
    dominant probability is exact.  Bound: the error of that arithmetic, restated in 64 bits with P and the result in
    fp16 and everything else exact, and 2 % for what the restatement leaves out (fp32 sums, scores at 2^-24)."""
    dev = cuda_or_skip()
    _lib, ops = _ops()
    heads, Lq = 20, 300
    gen = torch.Generator().manual_seed(L)
    q = h16(3 * torch.randn(1, Lq, heads * 64, generator=gen))
    kv = h16(torch.randn(1, L, 2 * heads * 64, generator=gen))
    y = ops.attention(q.half().to(dev), [kv.half().to(dev)], heads).cpu().double()
    _lib.device_status()
    split = lambda t: t.double().view(-1, heads, 64).transpose(0, 1)
    k, v = kv[0].chunk(2, dim=1)
    s = split(q[0]) @ split(k).transpose(1, 2) / 8 * 1.4426950408889634
    exact = torch.softmax(s * 0.6931471805599453, -1) @ split(v)
    m = s[..., :128].amax(-1, keepdim=True)
    top = s.amax(-1, keepdim=True)
    p = torch.exp2(s - torch.where(top > m + 8, top, m))
    model = ((p.half().double() @ split(v)) / p.sum(-1, keepdim=True)).half().double()
    err = lambda o: float((o - exact).norm() / exact.norm())
    got = err(split(y[0]))
    assert got <= 1.02 * err(model), f"{got:.4e} > 1.02 * {err(model):.4e}"


@pytest.mark.parametrize("keys,groups,split", PLANS)
@pytest.mark.parametrize("masked,total", [(1, 320), (63, 320), (64, 320), (65, 320), (128, 320), (129, 320), (200, 320), (319, 320), (320, 320), (70, 100), (100, 100)])
def test_attention_after_keys_of_minus_infinity(masked, total, keys, groups, split):
    """Keys whose scores are -inf (a mask feature, left padding) weigh nothing, however many come first; a row that has
    no other key is NaN."""
    dev = cuda_or_skip()
    _lib, ops = _ops()
    gen = torch.Generator().manual_seed(masked)
    q, kv = h16(torch.randn(1, 200, 128, generator=gen)), h16(torch.randn(1, total, 256, generator=gen))
    q[..., 5] = q[..., 70] = 1.0
    kv[0, :masked, 5] = kv[0, :masked, 70] = float("-inf")
    if split > -(-total // (keys or 64)):
        pytest.skip("more splits than key/value tiles")
    with _plan(keys, groups, split):
        y = ops.attention(q.half().to(dev), [kv.half().to(dev)], 2)
    if masked == total:
        assert torch.isnan(y).all()
    else:
        assert_close(y, po._sdpa_heads(q, kv[:, masked:], 2), what=f"{masked} keys of -inf first, split {split}")


@pytest.mark.parametrize("keys", [1, 15, 16, 17, 32, 33, 64, 65, 77, 112, 127, 128, 129])
@pytest.mark.parametrize("Lq,offset", [(1, 0), (128, 8), (129, 0), (300, 8)])
def test_attention_with_few_keys(keys, Lq, offset):
    """One slot of up to 128 keys in one pass, up to the first length that takes the general kernel: keys on, before and
    after a 16- and a 32-column boundary, ragged query tiles, output rows at 32-byte boundaries and between them."""
    dev = cuda_or_skip()
    _lib, ops = _ops()
    B, heads = 2, 3
    C = heads * 64
    gen = torch.Generator().manual_seed(keys + 1000 * Lq)
    q, kv = h16(torch.randn(B, Lq, C, generator=gen)), h16(torch.randn(B, keys, 2 * C, generator=gen))
    store = torch.full((B, Lq, C + 16), 7.0, dtype=torch.float16, device=dev)
    out = store[..., offset : offset + C]
    ops.attention(q.half().to(dev), [kv.half().to(dev)], heads, out=out)
    _lib.device_status()
    assert_close(out, po._sdpa_heads(q, kv, heads), what=f"attention of {keys} keys, Lq {Lq}")
    assert bool((store[..., :offset] == 7).all()) and bool((store[..., offset + C :] == 7).all())


def test_exponential_on_the_fma_pipe():
    """2^x by the polynomial: a relative error of at most 2.5e-7 (the bound of the special-function unit is 2^-22 =
    2.4e-7) wherever the result counts (x <= 8), as good as zero below -120, exactly one at zero, NaN, an odd count."""
    dev = cuda_or_skip()
    _lib, ops = _ops()
    x = torch.cat([torch.linspace(-30, 12, 200001), torch.arange(-110, 120).float(), torch.tensor([0.0, 0.5, -0.5, 126.4, -119.9])])
    limits = torch.tensor([-120.0, -200.0, -1e30, float("-inf"), float("nan")])
    xd = torch.cat([x, limits]).to(dev)
    assert xd.numel() % 2 == 1
    y = torch.full_like(xd, 7.0)
    l = _lib.lib()
    _lib.check(l.bxl_debug_exp2_f32(xd.data_ptr(), y.data_ptr(), xd.numel(), torch.cuda.current_stream().cuda_stream), l, kernels=0)
    y = y.cpu()
    ref = torch.exp2(x.double())
    assert float(((y[: x.numel()].double() - ref).abs() / ref).max()) <= 2.5e-7
    assert float(y[(x == 0).nonzero()[0, 0]]) == 1.0
    t = y[x.numel() :]
    assert bool((t[:4] >= 0).all()) and bool((t[:4] < 1e-35).all()) and bool(torch.isnan(t[4]))
