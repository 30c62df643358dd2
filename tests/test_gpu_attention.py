"""GPU parity of INT8 attention (difb200_attention_int8 / difb200_attention through the C-ABI)
against the CPU oracle.

Tier 1 (gated, the north star's bf16 bar: rel-L2 <= 2e-3, cosine >= 0.9999): kernel vs
orc_attention_int8, the CPU statement of the kernel's numerical contract on the same INT8 codes.
Tier 3 (gated with the reference's own bar for its INT8 attention, cosine >= 0.9999, reference
tests/owned_attention_tests.cpp:122-157): kernel vs the exact Attention of the reference CPU
executor (restated in orc_attention_exact, bit-identical to it)."""
import numpy as np
import pytest

import oracle_bridge as ob
from helpers import bf16_normal, cosine, from_torch_bf16, rel_l2, to_torch_bf16

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from diffusion_compiler_b200 import ops as _ops
    return _ops


def _qkv(rng, B, S, H, KV, D=128):
    """N(0,1) bf16 q/k/v, q and k RMS-normalised per token-head as a DiT block does."""
    one = ob.f32_to_bf16(np.ones(D, np.float32))
    q = ob.orc().rms_norm(bf16_normal(rng, (B, S, H, D)), one, 1e-6)
    k = ob.orc().rms_norm(bf16_normal(rng, (B, S, KV, D)), one, 1e-6)
    v = bf16_normal(rng, (B, S, KV, D))
    return q, k, v


def _check(ops, B, S, H, KV, masked, seed, q_gain=1.0):
    import torch
    rng = np.random.default_rng(seed)
    ob.orc().lib.orc_set_threads(8)
    q, k, v = _qkv(rng, B, S, H, KV)
    if q_gain != 1.0:
        q = ob.f32_to_bf16(ob.bf16_to_f32(q) * np.float32(q_gain))
    valid = None
    if masked:
        valid = np.ones((B, S), np.uint8)
        valid[:, max(0, S - max(1, S // 5)):] = 0  # the last fifth of the keys is padding
        valid[0, 0] = 0
    q8, qs = ob.orc().quantize_int8_rows([q.reshape(-1, 128)], 1)
    k8, ks = ob.orc().quantize_int8_rows([k.reshape(-1, 128)], 1)
    q8, k8 = q8.reshape(B, S, H, 128), k8.reshape(B, S, KV, 128)
    want = ob.orc().attention_int8(q8, qs, k8, ks, v, valid)
    t = lambda a: torch.from_numpy(a).cuda()
    tv = None if valid is None else t(valid)
    got = ops.attention_int8(t(q8), t(qs), t(k8), t(ks), to_torch_bf16(v), tv)
    got2 = ops.attention(to_torch_bf16(q), to_torch_bf16(k), to_torch_bf16(v), tv)
    torch.cuda.synchronize()
    ops.poll_status()
    g, g2, w = (ob.bf16_to_f32(from_torch_bf16(x)) if not isinstance(x, np.ndarray) else ob.bf16_to_f32(x)
                for x in (got, got2, want))
    assert np.isfinite(g).all()
    # quantising q/k on the GPU gives the same codes, hence the same output bits
    assert np.array_equal(from_torch_bf16(got), from_torch_bf16(got2))
    r, c = rel_l2(g, w), cosine(g, w)
    assert r <= 2e-3 and c >= 0.9999, "tier 1: rel-L2 %.3e cosine %.6f" % (r, c)
    if q_gain != 1.0:
        return r, c, None, None
    exact = ob.bf16_to_f32(ob.orc().attention_exact(q, k, v, valid))
    c3, r3 = cosine(g, exact), rel_l2(g, exact)
    assert c3 >= 0.9999, "tier 3: cosine vs exact attention %.6f (rel-L2 %.3e)" % (c3, r3)
    return r, c, r3, c3


@pytest.mark.parametrize("S", [1, 31, 128, 129, 300, 640])
def test_attention_int8_sizes(ops, S):
    _check(ops, 1, S, 2, 2, False, 10 + S)


@pytest.mark.parametrize("B,S,H,KV,masked", [(2, 384, 4, 4, True), (2, 300, 6, 2, True), (1, 520, 8, 1, False),
                                             (2, 257, 3, 3, True)])
def test_attention_int8_gqa_and_mask(ops, B, S, H, KV, masked):
    _check(ops, B, S, H, KV, masked, 77)


@pytest.mark.parametrize("B,S,H,KV,masked", [(1, 300, 2, 2, False), (2, 384, 4, 2, True)])
def test_attention_int8_running_maximum_path(ops, B, S, H, KV, masked):
    """Queries six times larger than a normalised block's: the score bound exceeds the limit of
    the fixed-maximum path, so the kernel keeps a running maximum and rescales its output (tier 1
    only: with logits this peaked the INT8 codes themselves move the exact result)."""
    _check(ops, B, S, H, KV, masked, 91, q_gain=6.0)


def test_attention_all_keys_masked_gives_zero(ops):
    import torch
    rng = np.random.default_rng(5)
    B, S, H, KV = 1, 200, 2, 2
    q, k, v = _qkv(rng, B, S, H, KV)
    valid = torch.zeros(B, S, dtype=torch.uint8, device="cuda")
    out = ops.attention(to_torch_bf16(q), to_torch_bf16(k), to_torch_bf16(v), valid)
    torch.cuda.synchronize()
    assert torch.count_nonzero(out.float()) == 0
    ops.poll_status()


def test_attention_repeatable(ops):
    """Two runs give identical bits (reference gate: repeat-bit-exact, owned_attention_tests.cpp:158-159)."""
    import torch
    rng = np.random.default_rng(6)
    q, k, v = _qkv(rng, 1, 1000, 4, 2)
    a = ops.attention(to_torch_bf16(q), to_torch_bf16(k), to_torch_bf16(v))
    b = ops.attention(to_torch_bf16(q), to_torch_bf16(k), to_torch_bf16(v))
    torch.cuda.synchronize()
    assert torch.equal(a.view(torch.int16), b.view(torch.int16))


@pytest.mark.parametrize("B,Sq,Sk,H,KV,masked,q_gain", [(1, 300, 1100, 4, 2, True, 1.0), (2, 256, 640, 2, 2, False, 1.0),
                                                        (1, 200, 900, 2, 1, True, 6.0)])
def test_attention_chunked_launches_match_the_single_launch(ops, B, Sq, Sk, H, KV, masked, q_gain):
    """The chunked form (keys taken in several launches that carry m, l and the fp32 outputs of
    every query row) against the single launch over all keys: in ring order as the token-sharded
    block consumes slices (own slice first, then the others, one group wrapping around the end of
    the key axis), also with the running-maximum path (q_gain 6). Powers of two scale exactly, so
    only the order of the fp32 sums may differ: rel-L2 <= 1e-4 here, far inside the path's bar."""
    import torch
    rng = np.random.default_rng(300 + Sk)
    q, _, _ = _qkv(rng, B, Sq, H, KV)
    _, k, v = _qkv(rng, B, Sk, H, KV)
    if q_gain != 1.0:
        q = ob.f32_to_bf16(ob.bf16_to_f32(q) * np.float32(q_gain))
    valid = None
    if masked:
        valid = np.ones((B, Sk), np.uint8)
        valid[:, 250:260] = 0          # a padded slice tail in the middle of the key axis
        valid[:, Sk - 37:] = 0
    q8, qs = ob.orc().quantize_int8_rows([q.reshape(-1, 128)], 1)
    k8, ks = ob.orc().quantize_int8_rows([k.reshape(-1, 128)], 1)
    t = lambda a: torch.from_numpy(a).cuda()
    args = (t(q8.reshape(B, Sq, H, 128)), t(qs), t(k8.reshape(B, Sk, KV, 128)), t(ks), to_torch_bf16(v))
    tv = None if valid is None else t(valid)
    whole = ops.attention_int8(*args, tv)
    tiles = (Sk + 127) // 128
    own = 2 if tiles > 3 else 1  # "this rank's slice" starts at tile `own`
    groups = [[(own, 1)], [(own + 1, tiles - own - 1), (0, 1)], [(1, own - 1)]] if own == 2 else \
             [[(own, 1)], [(own + 1, tiles - own - 1), (0, 1)]]
    groups = [[r for r in g if r[1] > 0] for g in groups]
    groups = [g for g in groups if g]
    parts = ops.attention_int8_chunked(*args, groups, tv)
    same_order = ops.attention_int8_chunked(*args, [[(0, 1)], [(1, tiles - 1)]], tv) if tiles > 1 else whole
    torch.cuda.synchronize()
    ops.poll_status()
    a, b, c = (ob.bf16_to_f32(from_torch_bf16(x)) for x in (parts, whole, same_order))
    assert np.isfinite(a).all()
    assert rel_l2(a, b) <= 1e-4 and cosine(a, b) >= 0.999999, (rel_l2(a, b), cosine(a, b))
    # same tile order as the single launch: the carried state continues the very same sums
    assert np.array_equal(from_torch_bf16(same_order), from_torch_bf16(whole)) or rel_l2(c, b) <= 1e-5


@pytest.mark.parametrize("size,grouping", [(2, ()), (4, ()), (8, ()), (8, (1, 2, 5)), (8, (1, 3, 4))])
def test_attention_launch_plans_of_every_rank_match_the_single_launch(ops, size, grouping):
    """The launch plan the token-sharded mode uses (difb200_world_plan: the own slice first, the other
    slices in the groups their ring steps arrive in, ranges that wrap around the end of the key
    axis) for every rank of a world of 2, 4 and 8, on one GPU: each rank's queries against the whole
    gathered key axis in its planned launches must equal the single launch over all keys."""
    import ctypes as C
    import torch
    from diffusion_compiler_b200 import _lib
    lib = _lib.lib()
    rng = np.random.default_rng(500 + size)
    H, KV, slice_tokens, local = 2, 2, 256, 200      # slices padded to 2 key tiles, 200 real tokens each
    Sk = size * slice_tokens
    _, k, v = _qkv(rng, 1, Sk, H, KV)
    valid = np.zeros((1, Sk), np.uint8)
    for r in range(size):
        valid[0, r * slice_tokens:r * slice_tokens + local] = 1
    k8, ks = ob.orc().quantize_int8_rows([k.reshape(-1, 128)], 1)
    t = lambda a: torch.from_numpy(a).cuda()
    keys = (t(k8.reshape(1, Sk, KV, 128)), t(ks), to_torch_bf16(v))
    for rank in range(size):
        q, _, _ = _qkv(rng, 1, local, H, KV)
        q8, qs = ob.orc().quantize_int8_rows([q.reshape(-1, 128)], 1)
        cap = 16
        ranges, first, count, n = (C.c_uint32 * (4 * cap))(), (C.c_int32 * cap)(), (C.c_int32 * cap)(), C.c_int32(0)
        sizes = (C.c_int32 * max(1, len(grouping)))(*grouping)
        assert lib.difb200_world_plan(rank, size, slice_tokens // 128, sizes, len(grouping), ranges, first, count, cap,
                                      C.byref(n)) == 0
        groups = [[(ranges[4 * i], ranges[4 * i + 1])] + ([(ranges[4 * i + 2], ranges[4 * i + 3])] if ranges[4 * i + 3] else [])
                  for i in range(n.value)]
        args = (t(q8.reshape(1, local, H, 128)), t(qs)) + keys
        whole = ops.attention_int8(*args, t(valid))
        parts = ops.attention_int8_chunked(*args, groups, t(valid))
        torch.cuda.synchronize()
        a, b = (ob.bf16_to_f32(from_torch_bf16(x)) for x in (parts, whole))
        # Another key order: the fp32 sums of the tensor cores round elsewhere, which moves about one
        # bf16 output in a thousand by one step (rel-L2 near 1e-4). A slice read twice, skipped or taken
        # from the wrong place would show as whole rows off by far more than one step.
        assert np.isfinite(a).all() and rel_l2(a, b) <= 3e-4, (size, rank, rel_l2(a, b))
        assert np.all(np.abs(a - b) <= 2.0 ** -7 * np.abs(b) + 1e-3 * np.abs(b).max()), (size, rank)
        assert np.mean(a != b) <= 0.01, (size, rank, float(np.mean(a != b)))
    ops.poll_status()


@pytest.mark.parametrize("B,Sq,Sk,H,KV,masked,q_gain", [
    (1, 700, 1100 + 3 * 512, 24, 8, True, 1.0),    # 72 items, 21 ragged tiles: two CTAs per item
    (2, 300, 1700, 12, 12, False, 1.0),            # 48 items of 14 tiles: three where their clusters fit
    (1, 130, 4096 + 77, 6, 2, True, 6.0),          # 6 items of 33 tiles: eight, running maximum
    (1, 1, 2048, 5, 5, True, 1.0),                 # one query row
    (1, 1400, 2500, 25, 25, False, 1.0),           # 150 items: one whole wave, then the rest split
])
def test_attention_split_over_keys_matches_the_plain_launch(ops, B, Sq, Sk, H, KV, masked, q_gain):
    """Items that would leave most SMs idle are split over the keys by clusters; the chunked form with one range is
    the same launch without the split. Powers of two scale exactly, so only the order of the fp32 sums differs:
    the bars of the launch plans above. The mask hides all keys of one CTA's share, and in the last entry of the
    batch all but one key."""
    import torch
    rng = np.random.default_rng(700 + Sk)
    q, _, _ = _qkv(rng, B, Sq, H, KV)
    _, k, v = _qkv(rng, B, Sk, H, KV)
    if q_gain != 1.0:
        q = ob.f32_to_bf16(ob.bf16_to_f32(q) * np.float32(q_gain))
    tv = None
    if masked:
        valid = np.ones((B, Sk), np.uint8)
        valid[:, :Sk // 2 + 200] = 0
        valid[:, Sk - 37:] = 0
        tv = torch.from_numpy(valid).cuda()
    q8, qs = ob.orc().quantize_int8_rows([q.reshape(-1, 128)], 1)
    k8, ks = ob.orc().quantize_int8_rows([k.reshape(-1, 128)], 1)
    t = lambda a: torch.from_numpy(a).cuda()
    args = (t(q8.reshape(B, Sq, H, 128)), t(qs), t(k8.reshape(B, Sk, KV, 128)), t(ks), to_torch_bf16(v))
    split = ops.attention_int8(*args, tv)
    again = ops.attention_int8(*args, tv)
    plain = ops.attention_int8_chunked(*args, [[(0, (Sk + 127) // 128)]], tv)
    torch.cuda.synchronize()
    ops.poll_status()
    assert torch.equal(split.view(torch.int16), again.view(torch.int16))
    a, b = (ob.bf16_to_f32(from_torch_bf16(x)) for x in (split, plain))
    assert np.isfinite(a).all() and rel_l2(a, b) <= 3e-4, rel_l2(a, b)
    assert np.all(np.abs(a - b) <= 2.0 ** -7 * np.abs(b) + 1e-3 * np.abs(b).max())
    assert np.mean(a != b) <= 0.01, float(np.mean(a != b))
    if masked:  # nothing valid anywhere: zeros
        none = ops.attention_int8(*args, torch.zeros_like(tv))
        assert torch.count_nonzero(none.float()) == 0


@pytest.mark.parametrize("case", ["share_masked", "bounds_apart", "bounds_apart_reversed"])
def test_attention_joins_key_ranges_whose_scores_are_far_below_their_maxima(ops, case):
    """Keys against their queries: every score is -50 or less in units of log2. In `share_masked` the first half of
    the keys is masked and the others score about -130, so a range without a valid key must not set a maximum.
    In the other two one key of one half scores -59 (a bound that the fixed maximum takes as +60) and all keys of the
    other half -69 (running maximum), which together outweigh it. The split, the plain and the chunked launches in
    both orders against the oracle, at the bar of the path (rel-L2 2e-3)."""
    import torch
    B, Sq, Sk, H, KV = 1, 130, 4096, 6, 2  # 6 items of 32 tiles: eight CTAs each
    rng = np.random.default_rng(11)
    half = Sk // 2
    q8 = np.full((B, Sq, H, 128), 100, np.int8) + rng.integers(-1, 2, (B, Sq, H, 128), dtype=np.int8)
    k8 = np.full((B, Sk, KV, 128), -100, np.int8)
    valid = np.ones((B, Sk), np.uint8)
    score = np.full((B, Sk, KV), -69.0)
    if case == "share_masked":
        k8 += rng.integers(-3, 4, k8.shape, dtype=np.int8)
        valid[:, :half] = 0
        score[:] = -130.0
    else:
        near = slice(0, half) if case == "bounds_apart" else slice(half, Sk)
        valid[:, near] = 0
        valid[:, near.start + 300] = 1
        score[:, near] = -59.0
    qs = np.full((B, Sq, H), 0.03, np.float32)
    unit = 128 * 100 * 100 * 0.03 / np.sqrt(128.0) * np.log2(np.e)  # what a key scale of 1 scores
    ks = (-score / unit).astype(np.float32)
    v = bf16_normal(rng, (B, Sk, KV, 128))
    want = ob.bf16_to_f32(ob.orc().attention_int8_rows(q8, qs.reshape(-1), k8, ks.reshape(-1), v, valid))
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    args = (t(q8), t(qs.reshape(-1)), t(k8), t(ks.reshape(-1)), to_torch_bf16(v))
    tiles = Sk // 128
    low, high = (0, tiles // 2), (tiles // 2, tiles // 2)
    got = {"split": ops.attention_int8(*args, t(valid)),
           "plain": ops.attention_int8_chunked(*args, [[(0, tiles)]], t(valid)),
           "low first": ops.attention_int8_chunked(*args, [[low], [high]], t(valid)),
           "high first": ops.attention_int8_chunked(*args, [[high], [low]], t(valid)),
           "single tiles": ops.attention_int8_chunked(*args, [[(i, 1)] for i in range(tiles)], t(valid))}
    torch.cuda.synchronize()
    ops.poll_status()
    for name, out in got.items():
        r = rel_l2(ob.bf16_to_f32(from_torch_bf16(out)), want)
        assert r <= 2e-3, (name, r)


@pytest.mark.parametrize("moved", ["q", "k", "both"])
def test_attention_takes_operands_that_start_on_two_bytes(ops, moved):
    """Contiguous bf16 q or k at an odd element offset goes through the general quantiser: the same bits."""
    import torch
    B, S, H, KV = 1, 300, 4, 2
    q, k, v = (to_torch_bf16(a) for a in _qkv(np.random.default_rng(8), B, S, H, KV))
    want = ops.attention(q, k, v)

    def shifted(a):
        return torch.empty(a.numel() + 1, dtype=a.dtype, device="cuda")[1:].view(a.shape).copy_(a)

    got = ops.attention(shifted(q) if moved != "k" else q, shifted(k) if moved != "q" else k, v)
    torch.cuda.synchronize()
    ops.poll_status()
    assert torch.equal(got.view(torch.int16), want.view(torch.int16))


@pytest.mark.parametrize("q_gain", [1.0, 6.0])
@pytest.mark.parametrize("Sq,tiles", [(130, 1), (130, 2), (256, 3), (130, 4), (257, 5), (130, 9)])
def test_attention_ring_and_query_tiles(ops, Sq, tiles, q_gain):
    """The two query tiles of a CTA run on their own and share the K/V ring, which also carries the query codes at the
    start and the outputs at the end: key tiles around the depth of the ring (4), a second query tile of one or two
    rows (it finishes first), keys whose first half is masked, with the fixed and the running maximum. Against the
    oracle at the bar of the path (rel-L2 2e-3); the same bits again."""
    import torch
    Sk = 128 * tiles - 5
    rng = np.random.default_rng(900 + tiles)
    q, _, _ = _qkv(rng, 1, Sq, 4, 2)
    _, k, v = _qkv(rng, 1, Sk, 4, 2)
    if q_gain != 1.0:
        q = ob.f32_to_bf16(ob.bf16_to_f32(q) * np.float32(q_gain))
    valid = np.ones((1, Sk), np.uint8)
    valid[:, :Sk // 2 + 11] = 0
    q8, qs = ob.orc().quantize_int8_rows([q.reshape(-1, 128)], 1)
    k8, ks = ob.orc().quantize_int8_rows([k.reshape(-1, 128)], 1)
    q8, k8 = q8.reshape(1, Sq, 4, 128), k8.reshape(1, Sk, 2, 128)
    want = ob.bf16_to_f32(ob.orc().attention_int8_rows(q8, qs, k8, ks, v, valid))
    t = lambda a: torch.from_numpy(a).cuda()  # noqa: E731
    args = (t(q8), t(qs), t(k8), t(ks), to_torch_bf16(v), t(valid))
    first, again = ops.attention_int8(*args), ops.attention_int8(*args)
    torch.cuda.synchronize()
    ops.poll_status()
    assert torch.equal(first.view(torch.int16), again.view(torch.int16))
    assert rel_l2(ob.bf16_to_f32(from_torch_bf16(first)), want) <= 2e-3


@pytest.mark.parametrize("exponent", [122, 100, -100])
@pytest.mark.parametrize("form", ["plain", "split", "chunked"])
def test_attention_running_maximum_with_large_and_small_values(ops, exponent, form):
    """No softmax weight is above 1, so values near the end of bf16's range stay finite where the maximum runs: V in
    [2^e, 2^(e+1)) under scores that rise by about a hundred powers of two along the keys, against the oracle on the same
    values without the power of two (rel-L2 2e-3, the bar of the path; the outputs themselves scale exactly)."""
    import torch
    rng = np.random.default_rng(31)
    Sq, Sk, H, KV = (130, 2048, 6, 2) if form == "split" else (130, 700, 4, 2)
    q = ob.f32_to_bf16(rng.standard_normal((1, Sq, H, 128)).astype(np.float32) * 8)
    k = rng.standard_normal((1, Sk, KV, 128)).astype(np.float32) * np.linspace(0.2, 3.0, Sk, dtype=np.float32)[:, None, None]
    v = ob.f32_to_bf16((1 + rng.random((1, Sk, KV, 128))).astype(np.float32))
    q8, qs = ob.orc().quantize_int8_rows([q.reshape(-1, 128)], 1)
    k8, ks = ob.orc().quantize_int8_rows([ob.f32_to_bf16(k).reshape(-1, 128)], 1)
    q8, k8 = q8.reshape(1, Sq, H, 128), k8.reshape(1, Sk, KV, 128)
    want = ob.bf16_to_f32(ob.orc().attention_int8_rows(q8, qs, k8, ks, v, np.ones((1, Sk), np.uint8)))
    scaled = ob.f32_to_bf16(ob.bf16_to_f32(v) * np.float32(2.0 ** exponent))
    t = lambda a: torch.from_numpy(a).cuda()  # noqa: E731
    args = (t(q8), t(qs), t(k8), t(ks), to_torch_bf16(scaled))
    tiles = (Sk + 127) // 128
    got = ops.attention_int8_chunked(*args, [[(0, 2)], [(2, tiles - 2)]]) if form == "chunked" else ops.attention_int8(*args)
    torch.cuda.synchronize()
    ops.poll_status()
    got = ob.bf16_to_f32(from_torch_bf16(got)).astype(np.float64)
    assert np.isfinite(got).all()
    assert rel_l2(got * 2.0 ** -exponent, want) <= 2e-3


@pytest.mark.parametrize("q_gain", [1.0, 6.0])
@pytest.mark.parametrize("masked", [False, True])
def test_attention_shows_every_score(ops, q_gain, masked):
    """Values that are one unit vector per key of one 128-key tile and zero elsewhere: output d of a query is the softmax
    weight of key d of that tile alone, so a score that was not made whole (or stood where another belongs) shows. Tile by
    tile, 72 CTAs, both query tiles, against the softmax in 64 bits: bf16 rounds a weight and the output once each (2^-8
    each), and the exponent's product and sum, at most 2^7 in fp32, move it by less than 2^-15."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(3)
    B, Sq, Sk, H, KV = 3, 257, 600, 12, 4
    q = torch.randn((B, Sq, H, 128), generator=g, device="cuda") * q_gain
    k = torch.randn((B, Sk, KV, 128), generator=g, device="cuda")
    q8, qs = ops.quantize_int8_rows([q.to(torch.bfloat16).view(-1, 128)], 1)
    k8, ks = ops.quantize_int8_rows([k.to(torch.bfloat16).view(-1, 128)], 1)
    q8, k8 = q8.view(B, Sq, H, 128), k8.view(B, Sk, KV, 128)
    valid = (torch.rand((B, Sk), generator=g, device="cuda") < 0.7).to(torch.uint8) if masked else None
    rep = lambda a: a.double().repeat_interleave(H // KV, 2)  # noqa: E731
    scores = torch.einsum("bqhd,bkhd->bhqk", q8.double() * qs.view(B, Sq, H, 1).double(),
                          rep(k8 * ks.view(B, Sk, KV, 1).double())) / 128 ** 0.5
    if masked:
        scores = scores.masked_fill(valid[:, None, None, :] == 0, -float("inf"))
    want = torch.softmax(scores, -1)
    for tile in range(0, Sk, 128):
        n = min(128, Sk - tile)
        v = torch.zeros((B, Sk, KV, 128), dtype=torch.bfloat16, device="cuda")
        v[:, tile:tile + n, :, :n] = torch.eye(n, dtype=torch.bfloat16, device="cuda")[None, :, None, :]
        out = ops.attention_int8(q8, qs, k8, ks, v, valid).double().permute(0, 2, 1, 3)[..., :n]
        w = want[..., tile:tile + n]
        assert bool(((out - w).abs() <= w * (2.0 ** -7 + 2.0 ** -10) + 1e-30).all()), tile
    ops.poll_status()


@pytest.mark.parametrize("rest", [40, 42, 43, 45])  # clusters of three behind a whole wave: one by one, all together from 43
def test_attention_split_where_its_clusters_fill_the_device(ops, rest):
    """The clusters behind a whole wave, started as SMs become free or together, against the same launch without a split
    (the bars of the split's test), back to back with new operands and the same bits again."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(rest)
    H, Sq, Sk = torch.cuda.get_device_properties(0).multi_processor_count + rest, 130, 2048
    v = torch.randn((1, Sk, 1, 128), generator=g, device="cuda").to(torch.bfloat16)
    runs = []
    for _ in range(2):
        q8, qs = ops.quantize_int8_rows([torch.randn((Sq * H, 128), generator=g, device="cuda").to(torch.bfloat16)], 1)
        k8, ks = ops.quantize_int8_rows([torch.randn((Sk, 128), generator=g, device="cuda").to(torch.bfloat16)], 1)
        args = (q8.view(1, Sq, H, 128), qs, k8.view(1, Sk, 1, 128), ks, v)
        runs.append((args, ops.attention_int8(*args), ops.attention_int8(*args)))
    for args, split, again in runs:
        plain = ops.attention_int8_chunked(*args, [[(0, Sk // 128)]])
        assert torch.equal(split.view(torch.int16), again.view(torch.int16))
        a, b = split.double(), plain.double()
        assert float((a - b).norm() / b.norm()) <= 3e-4
        assert float((a != b).double().mean()) <= 0.01
    ops.poll_status()


@pytest.mark.parametrize("q_gain", [1.0, 6.0])
@pytest.mark.parametrize("from_bf16", [False, True])
def test_attention_masks_at_the_edges_of_the_tables_segments(ops, q_gain, from_bf16):
    """Key masks against segments of 32 keys, whose first entry says whether any of them is masked: none, the first key
    alone, the last alone, all but the first, all; both builders of the key table. Against the contract, and the same
    bits as a call in which the masked keys' codes and values are others."""
    import torch
    rng = np.random.default_rng(17)
    B, S, H, KV = 2, 300, 2, 1
    q, k, v = _qkv(rng, B, S, H, KV)
    q = ob.f32_to_bf16(ob.bf16_to_f32(q) * np.float32(q_gain))
    valid = np.ones((B, S), np.uint8)
    valid[0, 32] = 0           # first of a segment
    valid[0, 95] = 0           # last of one
    valid[0, 129:160] = 0      # all but the first
    valid[0, 192:224] = 0      # a whole segment
    valid[1, 0] = 0
    valid[1, 255:] = 0
    q8, qs = ob.orc().quantize_int8_rows([q.reshape(-1, 128)], 1)
    k8, ks = ob.orc().quantize_int8_rows([k.reshape(-1, 128)], 1)
    q8, k8 = q8.reshape(B, S, H, 128), k8.reshape(B, S, KV, 128)
    want = ob.bf16_to_f32(ob.orc().attention_int8(q8, qs, k8, ks, v, valid))
    t = lambda a: torch.from_numpy(a).cuda()  # noqa: E731

    def run(k, v, k8, ks):
        if from_bf16:
            return ops.attention(to_torch_bf16(q), to_torch_bf16(k), to_torch_bf16(v), t(valid))
        return ops.attention_int8(t(q8), t(qs), t(k8), t(ks), to_torch_bf16(v), t(valid))

    got = run(k, v, k8, ks)
    assert rel_l2(ob.bf16_to_f32(from_torch_bf16(got)), want) <= 2e-3
    gone = valid == 0
    k2, v2 = k.copy(), v.copy()
    k2[gone], v2[gone] = ob.f32_to_bf16(np.float32([9.0]))[0], ob.f32_to_bf16(np.float32([-7.0]))[0]
    k82, ks2 = ob.orc().quantize_int8_rows([k2.reshape(-1, 128)], 1)
    assert torch.equal(run(k2, v2, k82.reshape(k8.shape), ks2).view(torch.int16), got.view(torch.int16))
    ops.poll_status()


@pytest.mark.parametrize("B,Sq,Sk,H,KV", [(1, 1, 77, 1, 1), (3, 513, 130, 6, 2), (2, 31, 5, 15, 5), (2, 257, 260, 7, 7), (5, 33, 128, 3, 1)])
def test_attention_items_of_every_batch_head_and_query_block(ops, B, Sq, Sk, H, KV):
    """The items of a launch against calls on one batch and head alone: the same bits. Rows whose sums are infinite, and
    rows of a batch without valid keys, stand among ordinary ones."""
    import torch
    rng = np.random.default_rng(B * Sq + Sk)
    q, k, v = _qkv(rng, B, Sq, H, KV)[0], *_qkv(rng, B, Sk, KV, KV)[1:]
    v[0, 0, 0, 5] = 0x7F80   # +infinity: this column of the heads that share it, the same rows' others as they are
    valid = np.ones((B, Sk), np.uint8)
    valid[B - 1] = 1 if B == 1 else 0
    (q8, qs), (k8, ks) = (ops.quantize_int8_rows([to_torch_bf16(x.reshape(-1, 128))], 1) for x in (q, k))
    q8, qs, k8, ks = q8.view(B, Sq, H, 128), qs.view(B, Sq, H), k8.view(B, Sk, KV, 128), ks.view(B, Sk, KV)
    tv, tm = to_torch_bf16(v), torch.from_numpy(valid).cuda()
    got = ops.attention_int8(q8, qs, k8, ks, tv, tm)
    for b in range(B):
        for h in range(H):
            g = h // (H // KV)
            mine = [x[b:b + 1, :, i:i + 1].contiguous() for x, i in ((q8, h), (qs, h), (k8, g), (ks, g), (tv, g))]
            alone = ops.attention_int8(*mine, tm[b:b + 1])
            assert torch.equal(got[b:b + 1, :, h:h + 1].contiguous().view(torch.int16), alone.view(torch.int16)), (b, h)
    assert torch.isposinf(got[0, :, :H // KV, 5]).all()
    ordinary = got.float().clone()
    ordinary[0, :, :H // KV, 5] = 0.0
    assert torch.isfinite(ordinary).all()
    if B > 1:
        assert torch.count_nonzero(got[B - 1]) == 0
    clean = v.copy()
    clean[0, 0, 0, 5] = 0
    rest = ops.attention_int8(q8, qs, k8, ks, to_torch_bf16(clean), tm).float()
    rest[0, :, :H // KV, 5] = 0.0
    assert torch.equal(ordinary, rest)
    ops.poll_status()


@pytest.mark.parametrize("masked", ["none", "first", "segment", "others", "random"])
def test_operands_of_few_and_of_many_rows_are_the_same(masked):
    """The operands' kernel takes two rows per lane where all its CTAs are resident at once and four else: one batch entry against the
    same entry four times, with masked keys on the edges of the key table's segments of 32 (its attention is not split)."""
    import torch
    from diffusion_compiler_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(3)
    tokens, heads = 300, 24
    q, k, v = (torch.randn((1, tokens, heads, 128), generator=g, device="cuda").to(torch.bfloat16) for _ in range(3))
    valid = torch.ones((1, tokens), dtype=torch.uint8, device="cuda")
    if masked == "first":
        valid[:, [0, 32, 160, 256]] = 0
    elif masked == "segment":
        valid[:, 64:96] = 0
    elif masked == "others":
        valid[:, [1, 31, 63, 95, 127, 130, 299]] = 0
    elif masked == "random":
        valid[:, torch.rand(tokens, generator=g, device="cuda") < 0.5] = 0
    key_valid = None if masked == "none" else valid
    one = ops.attention(q, k, v, key_valid=key_valid)
    four = ops.attention(*(t.repeat(4, 1, 1, 1) for t in (q, k, v)), key_valid=None if key_valid is None else valid.repeat(4, 1))
    torch.cuda.synchronize()
    ops.poll_status()
    assert bool(torch.isfinite(one.float()).all())
    assert all(torch.equal(four[i].view(torch.int16), one[0].view(torch.int16)) for i in range(4))
