"""GPU parity of the block-table GEMV users: fused sibling groups and the stacked-expert
SwitchGLU (decode and prefill paths), against the CPU oracle.  Tolerance 1e-3 relative L2 per
linear; the MoE chain (gate/up -> GLU -> down) is checked at 2e-3, as two roundings chain."""

from __future__ import annotations

import numpy as np
import pytest

from conftest import rel_err, synthetic_layer

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def cuda():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    return torch.device("cuda")


def _members(k, inf, outs, seed, cb=0):
    import ponyexl3_b200
    layers = []
    for i, o in enumerate(outs):
        tr, suh, svh, _ = synthetic_layer(k, inf, o, seed + i)
        layers.append(ponyexl3_b200.EXL3Layer(f"m{i}", inf, o, k, tr, suh, svh, None,
                                              mcg=(cb == 1), mul1=(cb == 2)))
    return layers


@pytest.mark.parametrize("rows", [1, 8, 16, 19])
@pytest.mark.parametrize("k,cb", [(4, 0), (3, 1), (6, 2)])
def test_fused_group_matches_members(cuda, oracle, rows, k, cb):
    """Rows {1, 8, 19} as the reference's group test (tests/test_exl3_fused.py:31-45)."""
    from ponyexl3_b200.fused import FusedEXL3Group

    layers = _members(k, 512, [512, 128, 256], seed=900 + k, cb=cb)
    grp = FusedEXL3Group(layers)
    x = np.random.default_rng(rows).standard_normal((rows, 512)).astype(np.float16)
    outs = grp.forward_all(torch.from_numpy(x).cuda())
    assert len(outs) == 3
    for o, l in zip(outs, layers):
        want = oracle.linear_forward(x, l.trellis, l.k, l.codebook_mode, l.suh, l.svh, None)
        assert o.shape == want.shape
        assert rel_err(o.cpu().numpy(), want) <= 1e-3


@pytest.mark.parametrize("dtype", ["float16", "bfloat16", "float32"])
@pytest.mark.parametrize("rows", [17, 24, 63])
def test_fused_group_with_scales_other_than_signs(cuda, oracle, rows, dtype):
    """suh holds fp16 multipliers, not only +-1: below 64 rows x * suh is not rounded before the rotation, for the
    members of a group (51, 72 and 189 rotated rows: both rotation kernels) as for a layer of its own.  The oracle
    rounds at the same places, so what is left is roundings of xh, y and sums that flip (1e-4); a rounded product
    would add its own 2^-12 rms, 2.8e-4 and more (5e-4 was seen)."""
    import ponyexl3_b200
    from ponyexl3_b200 import EXL3Linear
    from ponyexl3_b200.fused import FusedEXL3Group

    layers = []
    for i in range(3):
        tr, suh, svh, _ = synthetic_layer(4, 1024, 256, seed=970 + i)
        suh = (suh * np.random.default_rng(i).uniform(0.5, 1.5, 1024)).astype(np.float16)
        layers.append(ponyexl3_b200.EXL3Layer(f"m{i}", 1024, 256, 4, tr, suh, svh, None))
    xd = torch.from_numpy(np.random.default_rng(rows).standard_normal((rows, 1024)).astype(np.float32)).cuda().to(getattr(torch, dtype))
    x = xd.half().cpu().numpy()
    for o, l in zip(FusedEXL3Group(layers).forward_all(xd), layers):
        want = oracle.linear_forward(x, l.trellis, 4, 0, l.suh, l.svh, None)
        for got in (o, EXL3Linear(l)(xd)):
            assert rel_err(got.cpu().numpy(), want) <= 2.5e-4


@pytest.mark.parametrize("k,cb", [(4, 0), (3, 1), (6, 2)])
def test_block_tables_are_made_only_for_the_gemv(cuda, oracle, k, cb):
    """Up to 8 rows a group runs on the streamed GEMV over a block table; 9 and more take the GEMM, which has none,
    unless the scales are aligned for the GEMV (8 bytes) only."""
    from ponyexl3_b200 import EXL3Linear, EXL3MLPMonolith
    from ponyexl3_b200.fused import FusedEXL3Group

    layers = _members(k, 256, [256, 256], seed=980, cb=cb)
    grp = FusedEXL3Group(layers)
    mlp = EXL3MLPMonolith.from_fused_gate_up(grp, EXL3Linear(_members(4, 256, [128], seed=985)[0]))
    for rows in (9, 16, 17):
        x = np.random.default_rng(rows).standard_normal((rows, 256)).astype(np.float16)
        outs = grp.forward_all(torch.from_numpy(x).cuda())
        mlp(torch.from_numpy(x).cuda())
        assert not grp._tables
        for o, l in zip(outs, layers):
            assert rel_err(o.cpu().numpy(), oracle.linear_forward(x, l.trellis, k, cb, l.suh, l.svh, None)) <= 1e-3
    odd = torch.empty(grp._svh_cat.numel() + 8, dtype=torch.float16, device="cuda")
    odd[4:-4] = grp._svh_cat
    grp._svh_cat = odd[4:-4]
    for rows in (9, 12, 16):
        x = np.random.default_rng(rows).standard_normal((rows, 256)).astype(np.float16)
        for o, l in zip(grp.forward_all(torch.from_numpy(x).cuda()), layers):
            assert rel_err(o.cpu().numpy(), oracle.linear_forward(x, l.trellis, k, cb, l.suh, l.svh, None)) <= 1e-3
    mlp(torch.randn((8, 256), device="cuda").half())
    assert list(grp._tables) == [9, 12, 16, 8]


def test_fused_siblings_share_one_launch_and_refuse_bad_groups(cuda):
    from ponyexl3_b200.fused import FusedEXL3Group, fusable

    layers = _members(4, 256, [256, 128], seed=950)
    grp = FusedEXL3Group(layers)
    q, kproj = grp.sibling(0), grp.sibling(1)
    x = torch.randn((1, 256), device="cuda").half()
    a = q(x)
    assert grp._cache_x is x
    b = kproj(x)
    assert a.shape == (1, 256) and b.shape == (1, 128)
    assert list(grp.parameters()) == []
    bad = _members(4, 256, [256, 128], seed=951)
    bad[1].k = 5
    assert not fusable(bad)
    with pytest.raises(ValueError):
        FusedEXL3Group(bad)


def _experts(E, D, H, k, seed):
    rng = np.random.default_rng(seed)
    gu = rng.integers(0, 65536, size=(D // 16, E * 2 * H // 16, 16 * k), dtype=np.uint16)
    dn = rng.integers(0, 65536, size=(H // 16, E * D // 16, 16 * k), dtype=np.uint16)
    sg = lambda *s: np.where(rng.random(s) > 0.5, -1.0, 1.0).astype(np.float16)
    return dict(gu_trellis=gu, gu_suh=sg(E, 2, D), gu_svh=sg(E, 2 * H), dn_trellis=dn,
                dn_suh=sg(E, H), dn_svh=sg(E, D))


def _switch(w, k, cb, act="silu"):
    from ponyexl3_b200.moe import EXL3SwitchGLU

    t = {n: torch.from_numpy(np.ascontiguousarray(a).view(np.int16)).cuda() for n, a in w.items()}
    for n in ("gu_suh", "gu_svh", "dn_suh", "dn_svh"):
        t[n] = t[n].view(torch.float16)
    return EXL3SwitchGLU(**t, k=k, cb=cb, activation=act)


@pytest.mark.parametrize("tokens", [1, 3, 16])
@pytest.mark.parametrize("k,cb,act", [(4, 0, "silu"), (3, 1, "gelu")])
def test_switch_glu_decode_matches_oracle(cuda, oracle, tokens, k, cb, act):
    E, D, H, kk = 8, 256, 128, 2
    w = _experts(E, D, H, k, seed=40 + k)
    sw = _switch(w, k, cb, act)
    rng = np.random.default_rng(tokens)
    x = (rng.standard_normal((tokens, D)) * 0.5).astype(np.float16)
    idx = np.stack([rng.choice(E, size=kk, replace=False) for _ in range(tokens)]).astype(np.int64)
    y = sw(torch.from_numpy(x).cuda().view(1, tokens, D), torch.from_numpy(idx).cuda().view(1, tokens, kk))
    assert y.shape == (1, tokens, kk, D)
    want = oracle.switch_glu(x, idx, **w, k=k, cb=cb, activation=act)
    assert rel_err(y.cpu().numpy().reshape(tokens, kk, D), want) <= 2e-3


@pytest.mark.parametrize("k,tokens", [(4, 6), (4, 16), (1, 13), (6, 16)])
def test_switch_glu_few_tokens_by_expert(cuda, oracle, k, tokens):
    """Pairs that crowd on few experts: 6 tokens of 8 experts lie below the line between the two paths (48 - 8 < 55),
    13 and 16 above it (104 - 8, 128 - 8)."""
    E, D, H, kk = 8, 512, 512, 8
    w = _experts(E, D, H, k, seed=60 + k)
    rng = np.random.default_rng(tokens)
    x = (rng.standard_normal((tokens, D)) * 0.5).astype(np.float16)
    idx = np.stack([rng.permutation(E)[:kk] for _ in range(tokens)]).astype(np.int64)
    y = _switch(w, k, 0)(torch.from_numpy(x).cuda()[None], torch.from_numpy(idx).cuda()[None])
    want = oracle.switch_glu(x, idx, **w, k=k, cb=0)
    assert rel_err(y.cpu().numpy().reshape(tokens, kk, D), want) <= 2e-3


# K, tokens, experts, dims, top-k, and whether they go by expert (test_moe_plan.py checks that they do)
FEW_TOKENS = [
    (4, 6, 8, 512, 512, 8, False),
    (4, 16, 8, 512, 512, 8, True),
    (1, 13, 8, 512, 512, 8, True),
    (6, 16, 8, 512, 512, 8, True),
    (3, 16, 8, 640, 384, 8, True),
    (8, 16, 8, 512, 640, 8, True),
]


@pytest.mark.parametrize("k,tokens,E,D,H,kk,by_expert", FEW_TOKENS)
def test_switch_glu_few_tokens_on_both_sides_of_the_line(cuda, oracle, k, tokens, E, D, H, kk, by_expert):
    """Pairs that crowd on few experts, on both sides of the line between the two paths."""
    w = _experts(E, D, H, k, seed=60 + k)
    rng = np.random.default_rng(tokens)
    x = (rng.standard_normal((tokens, D)) * 0.5).astype(np.float16)
    idx = np.stack([rng.permutation(E)[:kk] for _ in range(tokens)]).astype(np.int64)
    y = _switch(w, k, 0)(torch.from_numpy(x).cuda()[None], torch.from_numpy(idx).cuda()[None])
    want = oracle.switch_glu(x, idx, **w, k=k, cb=0)
    assert rel_err(y.cpu().numpy().reshape(tokens, kk, D), want) <= 2e-3


def test_few_tokens_by_expert_do_not_grow_the_workspace(cuda, oracle):
    """Sixteen tokens on few experts fit the scratch that their way by pairs takes: a call captured behind a warm-up of one token
    must not allocate and clear a new workspace inside the graph."""
    from ponyexl3_b200 import _lib, ops

    dev = torch.cuda.current_device()
    old = ops.Workspace._per_device.pop(dev, None)
    if old is not None:
        ops.Workspace._retired.setdefault(dev, []).append(old)
    _lib.host().set_workspace(dev, 0, 0)
    E, D, H, kk = 8, 512, 512, 8
    w = _experts(E, D, H, 4, seed=97)
    sw = _switch(w, 4, 0)
    rng = np.random.default_rng(97)
    x = (rng.standard_normal((16, D)) * 0.5).astype(np.float16)
    idx = np.stack([rng.permutation(E)[:kk] for _ in range(16)]).astype(np.int64)
    xd, idd = torch.from_numpy(x).cuda()[None], torch.from_numpy(idx).cuda()[None]
    sw(xd[:, :1], idd[:, :1])
    before = ops.Workspace._per_device[dev]
    y = sw(xd, idd)
    assert ops.Workspace._per_device[dev] is before
    assert rel_err(y.cpu().numpy().reshape(16, kk, D), oracle.switch_glu(x, idx, **w, k=4, cb=0)) <= 2e-3


@pytest.mark.parametrize("name", ["_gu_svh", "_dn_svh"])
def test_few_tokens_with_scales_on_eight_bytes(cuda, oracle, name):
    """Output scales aligned for the GEMV only: sixteen tokens on few experts stay with it (the tile kernel refuses them)."""
    E, D, H, kk, T = 8, 512, 512, 8, 16
    w = _experts(E, D, H, 4, seed=95)
    sw = _switch(w, 4, 0)
    t = getattr(sw, name)
    odd = torch.empty(t.numel() + 8, dtype=t.dtype, device="cuda")[4:-4]
    odd.copy_(t.reshape(-1))
    setattr(sw, name, odd.view(t.shape))
    assert odd.data_ptr() % 16 == 8
    rng = np.random.default_rng(T)
    x = (rng.standard_normal((T, D)) * 0.5).astype(np.float16)
    idx = np.stack([rng.permutation(E)[:kk] for _ in range(T)]).astype(np.int64)
    y = sw(torch.from_numpy(x).cuda()[None], torch.from_numpy(idx).cuda()[None])
    assert rel_err(y.cpu().numpy().reshape(T, kk, D), oracle.switch_glu(x, idx, **w, k=4, cb=0)) <= 2e-3


def test_few_tokens_by_expert_keep_scales_unrounded(cuda, oracle):
    """Multipliers other than +-1: below 17 tokens x * suh is not rounded before the rotation on either path, so sixteen
    tokens at once are no further from the oracle than by fours (one row per pair).  Roundings that flip along the chain
    leave both 3e-4; a rounded product adds 2.8e-4 to 5e-4 in each of two projections, 1.6 times as much and more."""
    E, D, H, kk, T = 8, 512, 512, 8, 16
    w = _experts(E, D, H, 4, seed=90)
    rng = np.random.default_rng(7)
    for n in ("gu_suh", "dn_suh"):
        w[n] = (w[n] * rng.uniform(0.5, 1.5, w[n].shape)).astype(np.float16)
    x = (rng.standard_normal((T, D)) * 0.5).astype(np.float16)
    idx = np.stack([rng.permutation(E)[:kk] for _ in range(T)]).astype(np.int64)
    sw, xd, idd = _switch(w, 4, 0), torch.from_numpy(x).cuda()[None], torch.from_numpy(idx).cuda()[None]
    want = oracle.switch_glu(x, idx, **w, k=4, cb=0)
    err = lambda y: rel_err(y.cpu().numpy().reshape(T, kk, D), want)
    assert err(sw(xd, idd)) <= 1.25 * err(torch.cat([sw(xd[:, i:i + 4], idd[:, i:i + 4]) for i in range(0, T, 4)], 1))


def test_rows_of_x_read_once_for_all_their_copies(cuda):
    """Many rows: the rotation reads a row of x once for gate and up, or for all members of a group, and the result is what
    fewer rows give, whose copies are rotated one by one (16-row blocks x 128 columns below and above 64 per SM)."""
    from ponyexl3_b200 import EXL3Linear
    from ponyexl3_b200.fused import FusedEXL3Group

    E, D, H, kk = 16, 512, 128, 8
    sw = _switch(_experts(E, D, H, 4, seed=81), 4, 0)
    rng = np.random.default_rng(6)
    T = 4801
    x = torch.from_numpy((rng.standard_normal((T, D)) * 0.5).astype(np.float16)).cuda()
    idx = torch.from_numpy(np.stack([rng.permutation(E)[:kk] for _ in range(T)])).cuda()
    y = sw(x[None], idx[None])
    assert torch.equal(y, torch.cat([sw(x[None, i:i + 700], idx[None, i:i + 700]) for i in range(0, T, 700)], 1))
    layers = _members(4, 2048, [256, 128, 384], seed=82)
    x = torch.from_numpy(rng.standard_normal((9497, 2048)).astype(np.float32)).cuda().bfloat16()
    for got, l in zip(FusedEXL3Group(layers).forward_all(x), layers):
        want = EXL3Linear(l)(x)
        # the group's launch deals its tiles to other CTAs, whose fp32 sums are added in another order: some of the fp16
        # values that are rotated on the way out flip by an ulp (2^-11); a wrong row or multiplier would be of order 1
        assert rel_err(got.float().cpu().numpy(), want.float().cpu().numpy()) <= 2 ** -11


def test_switch_glu_prefill_matches_oracle_and_decode(cuda, oracle):
    E, D, H, kk, k = 8, 256, 128, 2, 4
    w = _experts(E, D, H, k, seed=77)
    sw = _switch(w, k, 0)
    rng = np.random.default_rng(5)
    T = 150
    x = (rng.standard_normal((T, D)) * 0.5).astype(np.float16)
    idx = np.stack([rng.choice(E, size=kk, replace=False) for _ in range(T)]).astype(np.int64)
    y = sw(torch.from_numpy(x).cuda().view(1, T, D), torch.from_numpy(idx).cuda().view(1, T, kk))
    want = oracle.switch_glu(x, idx, **w, k=k, cb=0)
    assert rel_err(y.cpu().numpy().reshape(T, kk, D), want) <= 2e-3


def test_config4_moe_block_one_token(cuda, oracle):
    """256 experts, top-8, hidden 2048, expert intermediate 512, K = 4: one token through router,
    stacked experts and weighted sum; expert outputs checked against the oracle."""
    from ponyexl3_b200.moe import EXL3MoEBlock, route_topk

    E, D, H, kk, k = 256, 2048, 512, 8, 4
    w = _experts(E, D, H, k, seed=4000)
    sw = _switch(w, k, 0)
    rng = np.random.default_rng(4001)
    # random trellis words decode to unit-variance weights: keep the chain inside fp16 range
    x = (rng.standard_normal((1, D)) * 0.02).astype(np.float16)
    logits = rng.standard_normal((1, E)).astype(np.float32)
    inds, scores = route_topk(torch.from_numpy(logits).cuda(), kk)
    assert abs(float(scores.sum()) - 1.0) < 1e-5
    y = sw(torch.from_numpy(x).cuda().view(1, 1, D), inds.view(1, 1, kk))
    want = oracle.switch_glu(x, inds.cpu().numpy(), **w, k=k, cb=0)
    assert rel_err(y.cpu().numpy().reshape(1, kk, D), want) <= 2e-3
    gate_w = torch.from_numpy(rng.standard_normal((E, D)).astype(np.float32) * 0.05).cuda()
    blk = EXL3MoEBlock(gate_w, sw, kk)
    out = blk(torch.from_numpy(x).cuda())
    assert out.shape == (1, D) and torch.isfinite(out.float()).all()


def test_config4_prefill_tile_table(cuda, oracle):
    """Config-4 expert dims with 128 tokens x top-8 = 1024 sorted pairs over 256 experts: most
    row tiles are ragged and many table slots stay unused."""
    E, D, H, kk, k = 256, 2048, 512, 8, 4
    w = _experts(E, D, H, k, seed=4100)
    sw = _switch(w, k, 0)
    rng = np.random.default_rng(4101)
    T = 128
    x = (rng.standard_normal((T, D)) * 0.02).astype(np.float16)
    idx = np.stack([rng.choice(E, size=kk, replace=False) for _ in range(T)]).astype(np.int64)
    y = sw(torch.from_numpy(x).cuda().view(1, T, D), torch.from_numpy(idx).cuda().view(1, T, kk))
    from ponyexl3_b200 import ops
    assert ops.Workspace.get(torch.device("cuda"), 1, 128).status() == 0
    want = oracle.switch_glu(x, idx, **w, k=k, cb=0)
    assert rel_err(y.cpu().numpy().reshape(T, kk, D), want) <= 2e-3


def test_config4_sixteen_tokens(cuda, oracle):
    """Config-4 dims with 16 tokens x top-8 = 128 (token, slot) pairs over about 100 distinct
    experts: the block-table GEMV with many blocks per CTA and a different sign vector per block."""
    from ponyexl3_b200 import ops
    from ponyexl3_b200.moe import route_topk

    E, D, H, kk, k, T = 256, 2048, 512, 8, 4, 16
    w = _experts(E, D, H, k, seed=4200)
    sw = _switch(w, k, 0)
    rng = np.random.default_rng(4201)
    x = (rng.standard_normal((T, D)) * 0.02).astype(np.float16)
    inds, _ = route_topk(torch.from_numpy(rng.standard_normal((1, T, E)).astype(np.float32)).cuda(), kk)
    y = sw(torch.from_numpy(x).cuda().view(1, T, D), inds.view(1, T, kk))
    assert ops.Workspace.get(torch.device("cuda"), 1, 128).status() == 0
    want = oracle.switch_glu(x, inds.reshape(T, kk).cpu().numpy(), **w, k=k, cb=0)
    assert rel_err(y.cpu().numpy().reshape(T, kk, D), want) <= 2e-3


def test_config4_4096_tokens_sampled(cuda, oracle):
    """Config-4 dims at 4096 tokens (32,768 pairs, full tile tables): every output row is finite
    and 256 sampled (token, slot) pairs match the oracle, each pair being independent of the rest."""
    from ponyexl3_b200 import ops
    from ponyexl3_b200.moe import route_topk

    E, D, H, kk, k, T = 256, 2048, 512, 8, 4, 4096
    w = _experts(E, D, H, k, seed=4300)
    sw = _switch(w, k, 0)
    rng = np.random.default_rng(4301)
    x = (rng.standard_normal((T, D)) * 0.02).astype(np.float16)
    inds, _ = route_topk(torch.from_numpy(rng.standard_normal((1, T, E)).astype(np.float32)).cuda(), kk)
    y = sw(torch.from_numpy(x).cuda().view(1, T, D), inds.view(1, T, kk))
    assert ops.Workspace.get(torch.device("cuda"), 1, 128).status() == 0
    y = y.cpu().numpy().reshape(T, kk, D)
    assert np.isfinite(y.astype(np.float32)).all()
    idx = inds.reshape(T, kk).cpu().numpy()
    toks = rng.choice(T, size=256, replace=False)
    slots = rng.integers(0, kk, size=256)
    want = oracle.switch_glu(x[toks], idx[toks, slots][:, None], **w, k=k, cb=0)[:, 0]
    assert rel_err(y[toks, slots], want) <= 2e-3


@pytest.mark.parametrize("k", [1, 4, 8])
@pytest.mark.parametrize("tokens,width", [(16, 2048), (16, 1920), (15, 2048)])
def test_decode_with_the_longest_ranges_rotates_in_the_kernel(cuda, k, tokens, width):
    """128 pairs give a GEMV half up to 56 rotated blocks, the most that are rotated inside the kernel: the same
    bits as with a rotation kernel of its own in front of it."""
    import torch
    from ponyexl3_b200 import _lib

    w = _experts(16, width, 512, k, seed=60 + k)
    m = _switch(w, k, 0)
    g = torch.Generator(device="cuda").manual_seed(k)
    x = (torch.randn((1, tokens, width), device="cuda", generator=g) * 0.02).half()
    idx = torch.topk(torch.randn((1, tokens, 16), device="cuda", generator=g), 8, dim=-1).indices
    got = m(x, idx).clone()
    _lib.load().exl3_tune_gemv(0, 0)
    try:
        want = m(x, idx).clone()
    finally:
        _lib.load().exl3_tune_gemv(0, 32 * 1024)
    assert torch.isfinite(got).all() and torch.equal(got, want)


@pytest.mark.parametrize("world", [2, 3, 8])
@pytest.mark.parametrize("tokens", [1, 5, 16])
def test_decode_over_an_expert_range_sums_to_the_full_switch(cuda, oracle, world, tokens):
    """Expert parallelism for few tokens, every rank's share computed one after the other on this
    GPU: a rank holds a contiguous expert range, the library picks its pairs on the device (the
    count never reaches the host) and leaves the other pairs' rows zero; the shares add up to the
    oracle's output, and a captured replay gives the same values."""
    from ponyexl3_b200 import ops
    from ponyexl3_b200.parallel import shard_expert_weights, shard_experts

    E, D, H, kk, k = 16, 256, 128, 4, 4
    w = _experts(E, D, H, k, seed=910 + world)
    rng = np.random.default_rng(tokens * 10 + world)
    x = (rng.standard_normal((tokens, D)) * 0.5).astype(np.float16)
    idx = np.stack([rng.choice(E, size=kk, replace=False) for _ in range(tokens)]).astype(np.int64)
    xd, idd = torch.from_numpy(x).cuda(), torch.from_numpy(idx).cuda()
    total = torch.zeros((tokens, kk, D), dtype=torch.float32, device="cuda")
    nonzero_rows = 0
    for rank in range(world):
        e0, e1 = shard_experts(E, world, rank)
        sw = _switch(shard_expert_weights(w, E, world, rank), k, 0)
        y = sw.decode_range(xd, idd, (e0, e1, E))
        held = (idd >= e0) & (idd < e1)
        assert bool((y[~held] == 0).all())                      # nobody else's rows are touched
        nonzero_rows += int(held.sum())
        if rank == 0:                                           # the same call from a CUDA graph
            stream = torch.cuda.Stream()
            with torch.cuda.stream(stream):
                sw.decode_range(xd, idd, (e0, e1, E))
                stream.synchronize()
                graph = torch.cuda.CUDAGraph()
                with torch.cuda.graph(graph, stream=stream):
                    yg = sw.decode_range(xd, idd, (e0, e1, E))
                graph.replay()
                stream.synchronize()
            assert torch.equal(yg, y)
        total += y.float()
    assert nonzero_rows == tokens * kk
    assert ops.Workspace.get(torch.device("cuda"), 1, 128).status() == 0
    want = oracle.switch_glu(x, idx, **w, k=k, cb=0)
    assert rel_err(total.cpu().numpy(), want) <= 2e-3


@pytest.mark.parametrize("world,act,T,kk", [(2, "silu", 96, 4), (4, "silu", 96, 4), (2, "gelu", 96, 4), (4, "gelu", 96, 4),
                                            (2, "silu", 20, 2)])
def test_prefill_over_an_expert_range_stores_rows_at_their_owners(cuda, oracle, world, act, T, kk):
    """Expert parallelism for many tokens, every rank's share computed one after the other on
    this GPU: tokens are partitioned (buffer p holds the output rows of partition p), a rank
    sorts and tiles only the pairs of its experts (their number stays on the device), its down
    projection stores each row into the owner's buffer and announces itself on every owner's
    counter.  After all ranks every counter holds `world` arrivals and the buffers hold the
    oracle's output."""
    import ctypes

    from ponyexl3_b200 import ops
    from ponyexl3_b200.parallel import shard_expert_weights, shard_experts

    E, D, H, k = 16, 256, 128, 4            # the last case: fewer than 64 pairs in all
    w = _experts(E, D, H, k, seed=930 + world)
    rng = np.random.default_rng(31 + world)
    x = (rng.standard_normal((T, D)) * 0.5).astype(np.float16)
    idx = np.stack([rng.choice(E, size=kk, replace=False) for _ in range(T)]).astype(np.int64)
    xd, idd = torch.from_numpy(x).cuda(), torch.from_numpy(idx).cuda()
    n_local = T // world * kk
    bufs = [torch.full((n_local, D), float("nan"), dtype=torch.float16, device="cuda") for _ in range(world)]
    ctrs = torch.zeros(world * 64, dtype=torch.int32, device="cuda")      # counters 256 bytes apart
    u64 = ctypes.c_uint64 * world
    y_ptrs = u64(*[b.data_ptr() for b in bufs])
    c_ptrs = u64(*[ctrs.data_ptr() + 256 * p for p in range(world)])
    for rank in range(world):
        e0, e1 = shard_experts(E, world, rank)
        sw = _switch(shard_expert_weights(w, E, world, rank), k, 0, act)
        sw.prefill_range(xd, idd, (e0, e1, E), (y_ptrs, c_ptrs, world, n_local, D))
    torch.cuda.synchronize()
    assert ctrs.view(world, 64)[:, 0].tolist() == [world] * world
    assert ops.Workspace.get(torch.device("cuda"), 1, 128).status() == 0
    got = torch.cat(bufs).cpu().numpy().reshape(T, kk, D)
    assert np.isfinite(got.astype(np.float32)).all()          # every row was written by somebody
    want = oracle.switch_glu(x, idx, **w, k=k, cb=0, activation=act)
    assert rel_err(got, want) <= 2e-3


@pytest.mark.parametrize("act", ["silu", "gelu"])
@pytest.mark.parametrize("rows", [1, 3, 8, 16])
def test_glu_folded_into_the_down_projection(cuda, oracle, act, rows):
    """EXL3_FLAG_GLU_*: the GEMV reads [gate | up] rows and applies the activation while loading —
    same result as the oracle's GLU (fp16 h) followed by its linear forward, for the fused
    rotation (few rows) and the rotation-kernel path (many rows)."""
    from ponyexl3_b200 import ops

    H, D, k, cb = 1024, 512, 4, 0
    tr, suh, svh, _ = synthetic_layer(k, H, D, seed=700 + rows)
    rng = np.random.default_rng(rows)
    gu = (rng.standard_normal((rows, 2 * H)) * 1.5).astype(np.float16)
    h = oracle.glu(gu[:, :H], gu[:, H:], act)
    want = oracle.linear_forward(h, tr, k, cb, suh, svh, None)
    t = lambda a: torch.from_numpy(a).cuda()
    y = ops.gemv(t(gu), t(tr.view(np.int16)), k, cb, t(suh), t(svh), None, glu=act)
    assert rel_err(y.cpu().numpy(), want) <= 1e-3
    assert ops.Workspace.get(torch.device("cuda"), 1, 128).status() == 0


def test_glu_on_load_equals_the_division_for_every_fp16_gate(cuda):
    """The quotient without a division inside the rotations against the activation kernel, which divides: the
    same bits for every finite fp16 gate.  Powers of two as `up` bring the products to unit size, which is exact."""
    from ponyexl3_b200 import ops

    H, k = 8192, 4
    tr, suh, svh, _ = synthetic_layer(k, H, 128, seed=710)
    t = lambda a: torch.from_numpy(a).cuda()
    g = torch.arange(65536, dtype=torch.int32).to(torch.int16).view(torch.float16).cuda()
    g = torch.where(g.isfinite(), g, torch.zeros_like(g))[torch.randperm(65536, generator=torch.Generator().manual_seed(1)).cuda()]
    size = (g.float() / (1 + torch.exp(-g.float()))).abs().clamp(2.0**-15, 2.0**14)
    up = torch.exp2(-torch.floor(torch.log2(size))).half()
    for rows in (8, 16):                                  # rotated inside the GEMV, and by the rotation kernel
        gu = torch.cat([g.view(8, H), up.view(8, H)], 1).repeat(rows // 8, 1)
        y = ops.gemv(gu, t(tr.view(np.int16)), k, 0, t(suh), t(svh), None, glu="silu")
        want = ops.gemv(ops.swiglu(gu), t(tr.view(np.int16)), k, 0, t(suh), t(svh), None)
        assert torch.isfinite(want).all() and torch.equal(y, want)


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("rows", [1, 12])
def test_glu_of_gates_beyond_the_range_of_fp16(cuda, dtype, rows):
    """Gates of bf16 and fp32 rows are not rounded to fp16 first: hugely negative ones give 0, in the rotation
    inside the GEMV and in the rotation kernel.  The same layer on the GLU's result computed outside: a gate whose
    exponential differs in the last bit flips one fp16 rounding of h, so the bound is that of a linear."""
    from ponyexl3_b200 import ops

    H, k = 512, 4
    tr, suh, svh, _ = synthetic_layer(k, H, 128, seed=720)
    t = lambda a: torch.from_numpy(a).cuda()
    gu = torch.from_numpy(np.random.default_rng(rows).standard_normal((rows, 2 * H)).astype(np.float32)).cuda().to(getattr(torch, dtype))
    gu[:, :32] = torch.tensor([-1e38, -3e34, -1e5, -95.0], device="cuda").repeat(8).to(gu.dtype)
    h = (gu[:, :H].float() / (1 + torch.exp(-gu[:, :H].float())) * gu[:, H:].float()).half()
    y = ops.gemv(gu, t(tr.view(np.int16)), k, 0, t(suh), t(svh), None, glu="silu")
    want = ops.gemv(h, t(tr.view(np.int16)), k, 0, t(suh), t(svh), None)
    assert (y.float() - want.float()).norm() / want.float().norm() < 1e-3


@pytest.mark.parametrize("rows", [1, 5, 16, 40])
def test_mlp_monolith_matches_the_three_linears(cuda, oracle, rows):
    """gate|up -> SiLU-GLU -> down as one module (the reference's EXL3MLPMonolith): equals the
    oracle's chain of linear forwards with h rounded to fp16 in between."""
    import ponyexl3_b200
    from ponyexl3_b200.fused import FusedEXL3Group
    from ponyexl3_b200.linear import EXL3Linear
    from ponyexl3_b200.mlp import EXL3MLPMonolith

    D, H, k = 512, 1024, 4
    gate, up = _members(k, D, [H, H], seed=1300)
    trd, suhd, svhd, _ = synthetic_layer(k, H, D, seed=1310)
    down = ponyexl3_b200.EXL3Layer("down", H, D, k, trd, suhd, svhd, None)
    mlp = EXL3MLPMonolith.from_fused_gate_up(FusedEXL3Group([gate, up]), EXL3Linear(down))
    x = (np.random.default_rng(rows).standard_normal((rows, D)) * 0.05).astype(np.float16)
    y = mlp(torch.from_numpy(x).cuda())
    g = oracle.linear_forward(x, gate.trellis, k, 0, gate.suh, gate.svh, None)
    u = oracle.linear_forward(x, up.trellis, k, 0, up.suh, up.svh, None)
    want = oracle.linear_forward(oracle.glu(g, u, "silu"), trd, k, 0, suhd, svhd, None)
    assert y.shape == (rows, D)
    assert rel_err(y.cpu().numpy(), want) <= 2e-3


@pytest.mark.parametrize("rows", [17, 64, 300])
@pytest.mark.parametrize("act", ["silu", "gelu"])
def test_group_and_mlp_prefill_equal_single_layers(cuda, rows, act):
    """More than 16 rows: the one GEMM of a group's members against each member alone (both rotation
    kernels, one and two token tiles), and the MLP against its linears and the activation."""
    from ponyexl3_b200.fused import FusedEXL3Group
    from ponyexl3_b200.linear import EXL3Linear
    from ponyexl3_b200.mlp import EXL3MLPMonolith
    from ponyexl3_b200.moe import glu

    x = torch.from_numpy(np.random.default_rng(rows).standard_normal((rows, 512)).astype(np.float32) * 0.05).cuda().bfloat16()
    layers = _members(4, 512, [384, 128, 640], seed=1400)
    for o, l in zip(FusedEXL3Group(layers).forward_all(x), layers):
        want = EXL3Linear(l)(x)
        assert o.shape == want.shape and o.is_contiguous()
        assert (o.float() - want.float()).norm() / want.float().norm() < 5e-4
    gate, up = _members(4, 512, [384, 384], seed=1410)
    down = EXL3Linear(_members(4, 384, [256], seed=1420)[0])
    y = EXL3MLPMonolith(FusedEXL3Group([gate, up]), down, activation=act)(x)
    want = down(glu(EXL3Linear(gate)(x), EXL3Linear(up)(x), act))
    assert (y.float() - want.float()).norm() / want.float().norm() < 1e-3
