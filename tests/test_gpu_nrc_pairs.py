"""The hash grid's paired gathers and scatters (corners x and x + 1 in one aligned
pair of entries) against the CPU oracle where they can go wrong: tables so small
that every index wraps, dense levels with even and odd rows, levels of one cell,
and samples on the box's faces, whose corners lie beyond the last cell.  The
bounds are those of bf16 activations and gradients, as for larger tables."""
import numpy as np
import pytest

import vrg
from nrc_ref import Model, corners

pytestmark = pytest.mark.gpu

LO, HI = (0.0, 0.0, 0.0), (64.0, 32.0, 64.0)


def _rel(a, b):
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-30))


@pytest.mark.parametrize("train", [0, vrg.NRC_TRAIN_WARP_MMA], ids=["tcgen05", "mma_sync"])
@pytest.mark.parametrize("levels,log2_t,base,top,n", [
    (1, 4, 1, 1, 1),
    (4, 4, 1, 16, 500),
    (5, 6, 1, 3, 500),
    (3, 10, 8, 10, 333),
    (16, 12, 2, 2048, 700),
])
def test_paired_corners_match_oracle(gpu_ctx, train, levels, log2_t, base, top, n):
    rng = np.random.default_rng(levels + n)
    c = vrg.RadianceCache(gpu_ctx, LO, HI, levels=levels, log2_table=log2_t, base_resolution=base, max_resolution=top,
                          batch=1024, learning_rate=1e-2, seed=3, flags=train)
    try:
        c.write(vrg.NRC_TABLE, (rng.normal(size=levels * (1 << log2_t) * 2) * 0.5).astype(np.float32))
        pos = rng.random((n, 3))
        edge = rng.random((n, 3))
        pos = np.where(edge < 0.1, 0.0, np.where(edge > 0.9, 1.0, pos))
        pos = (pos * np.array(HI)).astype(np.float32)
        nrm = np.zeros((n, 3), np.float32)
        nrm[np.arange(n), rng.integers(0, 3, n)] = 1.0
        d = rng.normal(size=(n, 3))
        d = (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)
        target = (np.abs(np.sin(pos[:, :1] * 0.2)) * np.array([[2.0, 1.0, 0.5]]) + 0.1).astype(np.float32)
        sc, dn, r1 = c.layout()
        m = Model(c.read(vrg.NRC_WEIGHTS), c.read(vrg.NRC_TABLE), levels, log2_t)
        yr = m.forward(corners(pos, LO, HI, sc, dn, r1, log2_t), nrm, d)
        assert _rel(c.query(pos, nrm, d), yr.detach().numpy()) < 2e-2
        c.write(vrg.NRC_ZERO_GRADS)
        c.train(pos, nrm, d, target, update=False)
        m.loss(yr, target).backward()
        got, ref = c.read(vrg.NRC_TABLE_GRADS), m.table.grad.numpy().reshape(-1)
        assert _rel(got, ref) < 5e-2
        assert not np.any(got[ref == 0])  # only the samples' corners have one
    finally:
        c.close()
