"""The CUDA trellis encoder (exl3_encode_tiles) through the C ABI: states bit-identical to the
reference's search (golden vectors) and to the oracle on random tiles, packed tiles that unpack
to the same states and decode to the codebook values of those states, and a whole matrix
quantised and decoded again."""

from __future__ import annotations

from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

GOLDEN = Path(__file__).resolve().parent / "golden" / "encoder.npz"


@pytest.fixture(scope="module")
def ops():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from ponyexl3_b200 import ops
    return ops


def _u16(t):
    return t.cpu().numpy().view(np.uint16)


def test_encoder_states_equal_the_reference(ops):
    g = np.load(GOLDEN)
    for i in range(int(g["n_cases"][0])):
        k, cb = int(g[f"c{i}_k"][0]), int(g[f"c{i}_cb"][0])
        states, packed = ops.quantize_tiles(torch.from_numpy(g[f"c{i}_w"]).cuda().view(1, 256), k, cb)
        assert (_u16(states)[0] == g[f"c{i}_states"]).all(), f"case {i}: K={k} cb={cb}"
        assert (_u16(ops.unpack_trellis(packed.view(1, 1, 16 * k), k))[0, 0] == g[f"c{i}_states"]).all()


@pytest.mark.parametrize("k,cb", [(2, 0), (3, 1), (4, 0), (4, 2)])
def test_encoder_matches_the_oracle_on_random_tiles(ops, oracle, k, cb):
    rng = np.random.default_rng(100 + 10 * k + cb)
    w = (rng.standard_normal((5, 256)) * rng.uniform(0.3, 2.0, size=(5, 1))).astype(np.float32)
    states, packed = ops.quantize_tiles(torch.from_numpy(w).cuda(), k, cb, max_tiles_in_flight=3)   # tiles share slots
    got = _u16(states)
    for t in range(5):
        want, _ = oracle.quantize_tile(w[t], k, cb)
        assert (got[t] == want).all(), f"tile {t}"
        assert (_u16(packed)[t] == oracle.pack_trellis_tile((want & ((1 << k) - 1)).astype(np.uint16), k)).all()


@pytest.mark.parametrize("k,cb", [(1, 0), (1, 2), (2, 1), (4, 1), (5, 2), (6, 0), (7, 1), (8, 0), (8, 2)])
def test_encoder_where_fp32_keys_cannot_decide(ops, oracle, k, cb):
    """Exact ties, weights that are codebook values, and magnitudes at which neighbouring costs are
    closer than fp32 resolves: every split of the bases over the threads takes the float64 path."""
    rng = np.random.default_rng(40 + k)
    w = rng.standard_normal((6, 256)).astype(np.float32)
    w[0] = 0.0
    w[1] = w[1].astype(np.float16).astype(np.float32)
    w[2] *= 1e4
    w[3] = np.sign(w[3]) * 0.5
    w[4] *= 1e-6
    states, packed = ops.quantize_tiles(torch.from_numpy(w).cuda(), k, cb)
    for t in range(6):
        want, _ = oracle.quantize_tile(w[t], k, cb)
        assert (_u16(states)[t] == want).all(), f"tile {t}"
        assert (_u16(packed)[t] == oracle.pack_trellis_tile((want & ((1 << k) - 1)).astype(np.uint16), k)).all()


@pytest.mark.parametrize("k,cb", [(1, 0), (2, 0), (3, 1), (4, 0), (5, 1), (6, 2), (7, 0), (8, 2)])
def test_encoder_of_weights_without_measure(ops, oracle, k, cb):
    """Squared errors of the size of the 1e30 that marks unreachable states and beyond the range of fp32, infinite
    weights and NaN, each at the start, in the middle and at the end of a tile: the states of the oracle's search."""
    rng = np.random.default_rng(60 + k)
    w = rng.standard_normal((11, 256)).astype(np.float32)
    w[0, 5] = 1e16
    w[1, 100] = np.nan
    w[2, 30] = np.inf
    w[3, 7] = -3e37
    w[4, [3, 200]] = 2e15, 5e15
    w[5, [0, 255]] = 4e17, 1e16
    w[6, [0, 128]] = np.nan, -np.inf
    w[7, 255] = np.nan
    w[9, ::5] = 9.9e12                                    # the largest weights of the ordinary search, one more beyond
    w[10, 17] = -1.1e13
    states, _ = ops.quantize_tiles(torch.from_numpy(w).cuda(), k, cb, max_tiles_in_flight=3)
    for t in range(11):
        want, _ = oracle.quantize_tile(w[t], k, cb)
        assert (_u16(states)[t] == want).all(), f"tile {t}"


@pytest.mark.parametrize("k,cb,max_pins", [(1, 2, 4), (2, 0, 4), (2, 2, 1), (3, 1, 0), (4, 0, 0), (4, 2, 4), (5, 0, 64), (6, 2, 0),
                                           (7, 2, 4), (8, 2, 4), (8, 0, 0)])
def test_encoder_free_and_pinned_paths(ops, oracle, k, cb, max_pins):
    """The searches that one pass over a tile answers, and the tiles it leaves to the search from the start: MUL1's thousand
    values tie at every third tile of K = 8, small multiples of one number tie nearly everywhere; no pinned pass, one, many."""
    rng = np.random.default_rng(200 + 10 * k + cb)
    w = rng.standard_normal((10, 256)).astype(np.float32)
    w[3] = np.round(w[3] * 4) / 4
    w[4, 64:] = 0.25
    w[5, :200] = 0.0
    states, packed = ops.quantize_tiles(torch.from_numpy(w).cuda(), k, cb, max_pins=max_pins, max_tiles_in_flight=7)
    for t in range(10):
        want, _ = oracle.quantize_tile(w[t], k, cb, max_pins)
        assert (_u16(states)[t] == want).all(), f"tile {t}"
        assert (_u16(packed)[t] == oracle.pack_trellis_tile((want & ((1 << k) - 1)).astype(np.uint16), k)).all()


@pytest.mark.parametrize("k,cb", [(1, 0), (1, 2), (2, 2), (4, 2), (8, 2)])
def test_encoder_of_tiles_it_leaves_early_and_of_large_weights(ops, oracle, k, cb):
    """Zeros, whose decisions are all ties: more than are noted, in the first steps or (a tile's front) in the last ones; weights far
    beyond the codebook; an ordinary tile behind them on the same slot."""
    w = np.random.default_rng(300 + k).standard_normal((6, 256)).astype(np.float32)
    w[0] = 0.0
    w[1, :3] = 0.0
    w[2, 128:] = 0.0
    w[3:5] *= 10.0
    states, _ = ops.quantize_tiles(torch.from_numpy(w).cuda(), k, cb, max_tiles_in_flight=1)
    for t in range(6):
        assert (_u16(states)[t] == oracle.quantize_tile(w[t], k, cb)[0]).all(), f"tile {t}"


@pytest.mark.parametrize("k,cb", [(3, 0), (4, 0), (6, 0), (6, 1)])
def test_encoder_where_first_errors_differ_below_the_total(ops, oracle, k, cb):
    """Codewords +a and -a in front of one path and a first weight of 1e-18 to 1e-15: both starts cost the same to the bit, but
    the search from the start sees the first error alone, and without a pinned pass its choice stays."""
    C = oracle.codebook_table(cb).astype(np.float64)
    G = C.reshape(1 << k, 1 << (16 - k))             # a column: the states with the same low bits
    a = np.abs(G).min(0)
    both = np.flatnonzero((G == a).any(0) & (G == -a).any(0) & (a > 0))
    tiles = []
    for seed in range(12):
        rng = np.random.default_rng(seed)
        w, s = np.zeros(256), int(rng.choice(both))
        w[0] = rng.choice([-1, 1]) * 10.0 ** rng.uniform(-18, -15)
        for t in range(1, 256):
            s = ((s << k) | int(rng.integers(1 << k))) & 0xFFFF
            w[t] = C[s] + rng.standard_normal() * 0.3 * 2.0 ** -k
        tiles.append(w.astype(np.float32))
    for max_pins in (0, 4):
        states, _ = ops.quantize_tiles(torch.from_numpy(np.stack(tiles)).cuda(), k, cb, max_pins=max_pins)
        for t, w in enumerate(tiles):
            assert (_u16(states)[t] == oracle.quantize_tile(w, k, cb, max_pins)[0]).all(), f"tile {t}"


def test_quantised_matrix_decodes_to_the_chosen_codebook_values(ops, oracle):
    k, cb = 3, 0
    rng = np.random.default_rng(3)
    inner = rng.standard_normal((32, 48)).astype(np.float32)
    trellis = ops.quantize_inner(torch.from_numpy(inner).cuda(), k, cb)
    assert tuple(trellis.shape) == (2, 3, 16 * k)
    w = ops.decode_packed_trellis(trellis, k, cb).float().cpu().numpy()
    assert w.shape == inner.shape
    assert float(((w - inner) ** 2).mean()) < 0.032            # the reference test's bound for K = 3
    # one tile against the oracle's search of the same tile in codeword order
    perm = oracle.tensor_core_perm()
    tile = inner[16:32, 16:32].reshape(256)[perm]
    _, decoded = oracle.quantize_tile(tile, k, cb)
    assert (w[16:32, 16:32].reshape(256)[perm] == decoded).all()
