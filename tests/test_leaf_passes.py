"""P2M, L2P, gather and unsort at the edges of their tiles: one state (summed
over lane groups), a few, the widest lane-group count below 17 states, one lane
per state from 17, two state blocks above 32; leaves of one, a few and more than
48 sources a group (shared by a CTA's warps), empty leaves; point counts beside a
multiple of the 32-point gather tile and one full tile.

Every multipole and local of the leaves enters the result, which is compared
with the FP64 oracle FMM of the same tree, order and identities.
"""

import numpy as np
import pytest

import cdfmm_b200
import oracle

pytestmark = pytest.mark.gpu

# Split BF16 in the M2L: 2^-16 of each product, 1.5e-5 of the far field, itself
# at most the total as no pair is close (a jittered lattice); doubled for the
# FP32 sums of the other passes.
REL = 3e-5


def lattice(side, rng):
    g = np.stack(np.meshgrid(*[np.arange(side)] * 3, indexing="ij"), axis=-1).reshape(-1, 3)
    return (g + 0.5 + rng.uniform(-0.1, 0.1, g.shape)) / side


def points(kind, n, rng):
    x = rng.permutation(lattice(11, rng))[:n]
    if kind == "dense":  # and one leaf of depth 2 with 512 more
        x = np.concatenate([x, 0.25 + 0.25 * lattice(8, rng)])
    return x


@pytest.mark.parametrize("order,K", [(0, 1), (2, 1), (6, 1), (3, 3), (6, 4), (5, 16), (4, 17), (6, 32), (3, 33), (8, 2)])
@pytest.mark.parametrize("kind,n", [("uniform", 31), ("uniform", 64), ("uniform", 1025), ("dense", 500)])
def test_leaf_passes_against_oracle(kind, n, order, K):
    rng = np.random.default_rng(1000 * order + 10 * K + n)
    x = points(kind, n, rng)
    box = {"root_centre": [0.5, 0.5, 0.5], "root_half_width": 0.5}
    m = rng.normal(size=(K, len(x), 3)).astype(np.float32)
    plan = cdfmm_b200.DevicePlan.from_points(x, order, 2, max_states=K, **box)
    plan.set_near_mode(cdfmm_b200.NEAR_FP32)  # with it the FP32 P2M
    out = plan.evaluate(m, output="both")
    plan.close()
    for k in sorted({0, K // 2, K - 1}):
        ref = oracle.fmm(x, x, m[k].astype(np.float64), order, 2, identities=np.arange(len(x)), **box)
        assert oracle.rel_l2(out["H"][k], ref["H"]) < REL
        assert oracle.rel_l2(out["phi"][k], ref["phi"]) < REL
