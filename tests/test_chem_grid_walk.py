"""The grid chemistry on inputs where no two claims compete, so that every result is
determined: positions, alive flags and counts equal the oracle's bit for bit.

* one e-aq (code 5, the lowest index) among H3O+: H3O+ do not react with each other, so
  which of them reacts is decided by the order of the walk alone;
* isolated pairs, at the edges of a warp and a block and in calls that share a captured
  schedule;
* the same beside more than 1024 radicals in one 1.5 nm cell (a step then walks the lists):
  OH-, which stay there, and H3O+, which spread.

Clusters are 2500 nm apart, 13 standard deviations of the widest pair's separation after
1 us."""
import ctypes as C

import numpy as np
import pytest

import oracle
from wgdna import _lib

EAQ, OH, H, H3O, OHM = 5, 0, 2, 3, 6
PAIRS = ((OH, OH), (OH, EAQ), (EAQ, EAQ), (EAQ, H3O), (EAQ, H), (H, H), (OH, H), (H3O, EAQ), (OH, OHM))


def sites(n, seed):
    """Cluster centres on a grid that leaves out the origin, at any place in their cells."""
    m = int(np.ceil((n + 1) ** (1 / 3)))
    k = np.arange(m) - m // 2
    c = np.stack(np.meshgrid(k, k, k), -1).reshape(-1, 3)
    c = c[np.any(c != 0, axis=1)]
    assert len(c) >= n
    return 2500.0 * c[:n] + np.random.default_rng(seed).uniform(0, 3, (n, 3))


def stars(n, partners, seed):
    g = np.random.default_rng(seed)
    c = sites(n, seed)
    first = np.concatenate([c, np.full((n, 1), EAQ)], axis=1)
    d = g.normal(size=(partners, n, 3))
    d *= (g.uniform(0, 0.45, (partners, n, 1)) / np.linalg.norm(d, axis=-1, keepdims=True))
    rest = np.concatenate([c[None] + d, np.full((partners, n, 1), H3O)], axis=-1).reshape(-1, 4)
    return np.ascontiguousarray(np.concatenate([first, rest]), np.float32)


def pairs(n, seed):
    """n radicals, two to a site; the last is alone when n is odd."""
    g = np.random.default_rng(seed)
    c = sites((n + 1) // 2, seed)
    code = np.array(PAIRS)[g.integers(0, len(PAIRS), len(c))]
    rad = np.empty((len(c), 2, 4))
    rad[:, :, :3] = c[:, None] + g.normal(0, 0.1, (len(c), 2, 3))
    rad[:, :, 3] = code
    return np.ascontiguousarray(rad.reshape(-1, 4)[:n], np.float32)


def crowd(code, n):
    return np.tile(np.array([[0.7, 0.8, 0.7, code]], np.float32), (n, 1))


def check(ctx, rad, seed):
    n = rad.shape[0]
    counts, pos, alive = oracle.chem_grid(rad, seed=seed)
    r = _lib.ChemGridResult()
    gp, ga = np.zeros((n, 4), np.float32), np.zeros(n, np.uint32)
    _lib.check("grid", _lib.lib().wgdna_chem_grid(ctx.h, _lib.ptr(rad), n, 16, 1000.0, seed, C.byref(r), _lib.ptr(gp),
                                                  _lib.ptr(ga), n))
    np.testing.assert_array_equal(np.array(r.counts), counts)
    np.testing.assert_array_equal(ga != 0, np.asarray(alive).reshape(-1) != 0)
    np.testing.assert_array_equal(gp.view(np.uint32), np.ascontiguousarray(pos, np.float32).reshape(n, 4).view(np.uint32))
    return counts


@pytest.mark.gpu
@pytest.mark.parametrize("partners", [2, 5, 12, 60])
def test_order_of_the_walk(ctx, partners):
    """Up to 60 contacts of one radical: more than it keeps at a time."""
    counts = check(ctx, stars(400, partners, partners), 11)
    assert counts[-1][2] > 200                       # H made


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 2, 31, 33, 255, 256, 257, 511, 512, 513, 4096])
def test_isolated_pairs(ctx, n):
    check(ctx, pairs(n, n), 7)


@pytest.mark.gpu
def test_schedule_of_another_size_and_key(ctx):
    """4097 to 4350 radicals share one captured schedule, 255 have their own."""
    for n, seed in ((4350, 3), (4097, 3), (4350, 4), (255, 5), (4200, 6 + (5 << 40))):
        check(ctx, pairs(n, n), seed)


@pytest.mark.gpu
@pytest.mark.parametrize("code,n", [(OHM, 1100), (H3O, 1500)])
def test_beside_an_overfull_cell(ctx, code, n):
    """OH- keep their cell overfull in every step.  Of the H3O+, half start displaced by 0.46 nm
    per axis: about 1290 are in the cell at first, and after 1 ns they have left it."""
    rad = np.concatenate([pairs(1500, 8), crowd(code, n)])
    check(ctx, rad, 21)
    check(ctx, pairs(1500, 9), 22)                   # lists and tables are left empty
