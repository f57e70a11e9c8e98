"""GPU parity of the tensor-core prefill GEMM (rows > 16) through the module and the C ABI,
against the CPU oracle.  Tolerance: relative L2 error <= 1e-3 (fp32 accumulate)."""

from __future__ import annotations

import numpy as np
import pytest

from conftest import rel_err, synthetic_layer

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

REL_TOL = 1e-3


@pytest.fixture(scope="module")
def mod():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    import ponyexl3_b200
    from ponyexl3_b200 import ops
    from ponyexl3_b200.linear import EXL3Linear

    class NS:
        pass

    ns = NS()
    ns.ops, ns.EXL3Linear, ns.EXL3Layer = ops, EXL3Linear, ponyexl3_b200.EXL3Layer
    return ns


def _layer(mod, k, inf, outf, seed, cb=0, bias=False):
    tr, suh, svh, b = synthetic_layer(k, inf, outf, seed, bias=bias)
    return mod.EXL3Layer("test", inf, outf, k, tr, suh, svh, b, mcg=(cb == 1), mul1=(cb == 2))


def _check(mod, oracle, layer, x):
    m = mod.EXL3Linear(layer)
    y = m(torch.from_numpy(x).cuda()).cpu().numpy()
    want = oracle.linear_forward(x.astype(np.float16), layer.trellis, layer.k, layer.codebook_mode,
                                 layer.suh, layer.svh, layer.bias)
    assert y.shape == want.shape and y.dtype == np.float16
    assert np.isfinite(y.astype(np.float32)).all()
    e = rel_err(y, want)
    assert e <= REL_TOL, f"rel err {e}"
    assert mod.ops.Workspace.get(torch.device("cuda"), 1, 128).status() == 0


@pytest.mark.parametrize("k", range(1, 9))
@pytest.mark.parametrize("cb", [0, 1, 2])
def test_gemm_all_k_all_codebooks(mod, oracle, k, cb):
    layer = _layer(mod, k, 256, 384, seed=500 + 10 * k + cb, cb=cb, bias=(k % 2 == 1))
    x = np.random.default_rng(k).standard_normal((40, 256)).astype(np.float16)
    _check(mod, oracle, layer, x)


@pytest.mark.parametrize("k,cb,bias", [(4, 0, False), (2, 1, True), (5, 2, False), (8, 0, True), (1, 0, False)])
@pytest.mark.parametrize("rows,inf,outf", [(1024, 256, 256), (1500, 512, 384), (2049, 128, 640)])
def test_gemm_many_rows(mod, oracle, rows, inf, outf, k, cb, bias):
    """Several tiles of tokens, whole and ragged, two to five column tiles, two to eight k-steps."""
    layer = _layer(mod, k, inf, outf, seed=7000 + rows + k, cb=cb, bias=bias)
    x = np.random.default_rng(rows + k).standard_normal((rows, inf)).astype(np.float16)
    _check(mod, oracle, layer, x)


@pytest.mark.parametrize("rows", [17, 128, 129, 256, 300, 513])
def test_gemm_ragged_row_counts(mod, oracle, rows):
    layer = _layer(mod, 4, 512, 256, seed=77)
    x = np.random.default_rng(rows).standard_normal((rows, 512)).astype(np.float16)
    _check(mod, oracle, layer, x)


@pytest.mark.parametrize("rows,inf,outf,k,cb", [
    (17, 4096, 128, 4, 0),      # one output tile shared by many CTAs
    (40, 2048, 384, 3, 2),      # shared tiles, tokens not a multiple of 32
    (250, 1024, 256, 8, 0),     # K = 8: fewer tokens per tile fit the activation ring, two token tiles
    (257, 1152, 128, 7, 1),     # one row more than a tile, a k-range that is no multiple of the ring
    (700, 128, 640, 1, 0),      # two k-steps per tile, whole tiles
    (272, 512, 128, 4, 0),      # two token tiles of 144 and 128
    (384, 640, 256, 3, 0),      # two of 192
    (336, 1024, 128, 8, 2),     # two at K = 8
    (400, 512, 256, 5, 1),      # two, the second a few tokens short
    (1537, 256, 384, 6, 0),     # a last tile of few tokens
])
def test_gemm_tiles_shared_between_ctas(mod, oracle, rows, inf, outf, k, cb):
    layer = _layer(mod, k, inf, outf, seed=rows, cb=cb, bias=rows % 2 == 0)
    x = np.random.default_rng(rows).standard_normal((rows, inf)).astype(np.float16)
    _check(mod, oracle, layer, x)
    m = mod.EXL3Linear(layer)
    xd = torch.from_numpy(x).cuda()
    first = m(xd)
    assert all(torch.equal(m(xd), first) for _ in range(3))      # whoever finishes a shared tile
    assert mod.ops.Workspace.get(torch.device("cuda"), 1, 128).status() == 0


@pytest.mark.parametrize("rows", [9, 16, 33, 100, 128])
@pytest.mark.parametrize("inf,outf,k,cb", [
    (2048, 384, 4, 0),          # eight CTAs of four k-steps per tile; more CTAs than pieces of 16 tokens, and as many
    (2048, 2560, 5, 1),         # seven
    (1152, 5120, 3, 2),         # three
    (896, 8192, 8, 0),          # two, the deepest packed tiles
])
def test_gemm_tiles_of_clusters(mod, oracle, rows, inf, outf, k, cb):
    """The CTAs of a tile as a cluster that shares out its tokens: repeatable, and nothing left behind in shared memory."""
    layer = _layer(mod, k, inf, outf, seed=rows + inf, cb=cb, bias=rows % 2 == 1)
    x = np.random.default_rng(rows).standard_normal((rows, inf)).astype(np.float16)
    _check(mod, oracle, layer, x)
    m = mod.EXL3Linear(layer)
    xd = torch.from_numpy(x).cuda()
    first = m(xd)
    assert all(torch.equal(m(xd), first) for _ in range(3))


# Clusters of each size, by rows (test_gemm_plan.py checks that the plan takes them): where the exchanged sums are largest, at
# 113 to 128 tokens a tile, and where the packed tiles are.
CLUSTERS = [
    (1792, 1024, 4, 1, 77, 7),
    (1792, 1024, 4, 0, 128, 6),
    (1792, 1024, 5, 2, 121, 5),
    (1536, 1024, 6, 0, 100, 5),
    (1536, 1024, 6, 0, 90, 6),
    (1792, 1024, 7, 0, 113, 4),
    (1920, 2048, 7, 1, 128, 4),
    (1792, 1024, 7, 2, 256, 4),         # two tiles of tokens
    (1792, 1024, 8, 2, 112, 7),
    (1792, 1024, 8, 0, 128, 4),
    (1920, 2048, 8, 1, 120, 4),
    (4096, 1024, 8, 0, 128, 8),         # two stages of activations
    (4096, 1024, 8, 2, 9, 8),
]


@pytest.mark.parametrize("inf,outf,k,cb,rows,n", CLUSTERS)
def test_gemm_clusters_beside_the_rings(mod, oracle, inf, outf, k, cb, rows, n):
    layer = _layer(mod, k, inf, outf, seed=rows + inf + k, cb=cb, bias=rows % 2 == 1)
    x = np.random.default_rng(rows).standard_normal((rows, inf)).astype(np.float16)
    _check(mod, oracle, layer, x)
    m = mod.EXL3Linear(layer)
    xd = torch.from_numpy(x).cuda()
    first = m(xd)
    assert all(torch.equal(m(xd), first) for _ in range(3))
    assert mod.ops.Workspace.get(torch.device("cuda"), 1, 128).status() == 0


# Shapes of each form of the kernel (test_gemm_plan.py checks that the plan takes it): tiles of more than the
# ordinary number of tokens, whose MMAs are two halves; two and more ordinary tiles per CTA; hardly more than one.
FORMS = [
    (257, 128, 9600, 4, 0, "wide"),     # the smallest wide tile, halves of 144 and 128 tokens
    (384, 128, 9600, 4, 1, "wide"),     # the largest
    (384, 128, 9600, 1, 2, "wide"),
    (368, 128, 9600, 5, 0, "wide"),     # the largest at K = 5 to 8
    (225, 128, 9600, 6, 1, "wide"),
    (352, 128, 9600, 7, 2, "wide"),
    (193, 128, 9600, 8, 0, "wide"),     # halves of 112 and 96, the second ragged
    (336, 128, 9600, 8, 1, "wide"),
    (760, 128, 6400, 4, 0, "wide"),     # two wide tiles of tokens
    (4625, 128, 1024, 4, 0, "wide"),    # a last tile of one token: its second half is empty
    (3552, 128, 1024, 8, 2, "wide"),    # a last tile of sixteen
    (256, 256, 38400, 4, 0, "ahead"),   # two ordinary tiles per CTA and more
    (17, 256, 38400, 3, 2, "ahead"),
    (40, 256, 384, 4, 0, "plain"),
    (300, 256, 384, 8, 1, "plain"),
]


@pytest.mark.parametrize("rows,inf,outf,k,cb,form", FORMS)
def test_gemm_forms(mod, oracle, rows, inf, outf, k, cb, form):
    layer = _layer(mod, k, inf, outf, seed=rows + k, cb=cb, bias=rows % 2 == 0)
    x = np.random.default_rng(rows).standard_normal((rows, inf)).astype(np.float16)
    _check(mod, oracle, layer, x)


def test_gemm_of_many_tiles_per_cta_equals_small_calls(mod):
    """Every CTA has several tiles and decodes ahead of the one it finishes: the same rows in calls of 128
    (one tile per CTA) and all at once, several times over."""
    m = mod.EXL3Linear(_layer(mod, 4, 5120, 5120, seed=81))
    x = torch.from_numpy(np.random.default_rng(8).standard_normal((2048, 5120)).astype(np.float16)).cuda()
    want = torch.cat([m(x[i:i + 128]) for i in range(0, 2048, 128)]).float()
    for _ in range(6):
        y = m(x).float()
        assert (y - want).abs().max() < 0.02 * want.abs().mean() and (y - want).norm() / want.norm() < 5e-4


def test_gemm_many_tiles_and_k_steps(mod, oracle):
    """More tiles than one wave of k-steps per stage ring, several tiles per CTA."""
    layer = _layer(mod, 4, 2048, 1280, seed=78, bias=True)
    x = np.random.default_rng(5).standard_normal((600, 2048)).astype(np.float16)
    _check(mod, oracle, layer, x)


def test_gemm_bf16_activations(mod, oracle):
    layer = _layer(mod, 4, 512, 512, seed=79)
    xb = torch.from_numpy(np.random.default_rng(6).standard_normal((200, 512)).astype(np.float32)).cuda().to(torch.bfloat16)
    y = mod.EXL3Linear(layer)(xb).cpu().numpy()
    want = oracle.linear_forward(xb.float().cpu().numpy().astype(np.float16), layer.trellis, 4, 0,
                                 layer.suh, layer.svh, None)
    assert rel_err(y, want) <= REL_TOL


def test_gemm_matches_gemv_rows(mod):
    """The two kernels implement one contract: the same rows through either agree."""
    layer = _layer(mod, 5, 1024, 768, seed=80, bias=True)
    m = mod.EXL3Linear(layer)
    x = torch.from_numpy(np.random.default_rng(7).standard_normal((64, 1024)).astype(np.float16)).cuda()
    big = m(x)
    small = torch.cat([mod.ops.gemv(x[i:i + 16], m._trellis, 5, 0, m._suh, m._svh, m._bias) for i in range(0, 64, 16)])
    assert (big.float() - small.float()).norm() / small.float().norm() < 5e-4


def test_config3_prefill_shape_sampled(mod, oracle):
    """M = 8192 tokens x 5120 -> 5120, K = 4, 3INST, bf16 activations: full run on the GPU,
    512 sampled rows checked against the oracle (the oracle's decode is shared)."""
    layer = _layer(mod, 4, 5120, 5120, seed=3000)
    rng = np.random.default_rng(3001)
    xb = torch.from_numpy(rng.standard_normal((8192, 5120)).astype(np.float32)).cuda().to(torch.bfloat16)
    y = mod.EXL3Linear(layer)(xb)
    assert mod.ops.Workspace.get(torch.device("cuda"), 1, 128).status() == 0
    idx = np.sort(rng.choice(8192, size=512, replace=False))
    xs = xb[torch.from_numpy(idx).cuda()].float().cpu().numpy().astype(np.float16)
    w = oracle.decode_packed_trellis(layer.trellis, 4, 0)
    want = oracle.linear_forward(xs, layer.trellis, 4, 0, layer.suh, layer.svh, None, w=w)
    assert rel_err(y[torch.from_numpy(idx).cuda()].cpu().numpy(), want) <= REL_TOL
