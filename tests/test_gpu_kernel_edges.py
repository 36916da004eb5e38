"""Kernels at the sizes where their tiling can go wrong: edges of tiles, remainders, the smallest and the
largest of a range."""
import numpy as np
import pytest

import oracle
from nrltb import KMesh, synth

pytestmark = pytest.mark.gpu


def _atoms(n, basis, seed):
    """n displaced atoms of one species in a row of simple cubic cells."""
    st = synth.supercell(synth.SC_BASIS, 4.6, (n, 1, 1), lambda b: 1, 0.1, np.random.default_rng(seed))
    return st, synth.make_params([basis], [4.0], synth.PARAM_SEED)


@pytest.mark.parametrize("natoms,basis", [(1, 1), (1, 9), (8, 4), (11, 9), (7, 9), (16, 4)])
@pytest.mark.parametrize("nk", [1, 3, 4, 5, 9])
def test_bloch_sums_over_k_groups_and_tiles(ctx, natoms, basis, nk):
    """H and S of every k: matrix orders 1, 9, 32, 99, 63, 64 against tiles of 32, k lists around groups of 4.
    Each element is a sum of at most a few hundred FP64 products in the oracle's order: 1e-13 of the largest."""
    st, par = _atoms(natoms, basis, 5)
    km = KMesh(np.random.default_rng(nk).uniform(-0.5, 0.5, (nk, 3)), np.full(nk, 1.0 / nk))
    for which in (0, 1):
        got = ctx.setham(st, par, km, which)
        want = oracle.setham(st, par, km, which)
        for g, o in zip(got, want):
            assert np.abs(g - o).max() <= 1e-13 * max(np.abs(o).max(), 1e-300)
