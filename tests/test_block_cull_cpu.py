"""The tile-8 and tile-4 kernels evaluate a Gaussian on a 4^3 block only if no separating plane rules
the block out (``plane_threshold`` in gsv_common.cuh, ``plane_separates`` in gsv_render.cu).  The
rule restated in float32: no block it rules out may hold a voxel that the row form of the quadratic,
within its own rounding of the exact one, could include (m <= 9 (1 + 8.3e-4))."""
import numpy as np
import pytest

F = np.float32


def _threshold(q):
    q00, h01, h02, q11, h12, q22 = q.T
    with np.errstate(all="ignore"):
        i0, i1, i2 = F(1) / q00, F(1) / q11, F(1) / q22
        r01, r02, r12 = h01 * h01 * i0 * i1, h02 * h02 * i0 * i2, h12 * h12 * i1 * i2
        det = F(1) + F(2) * (h01 * i0) * (h02 * i2) * (h12 * i1) - r01 - r02 - r12
        ok = ((q.T[[0, 3, 5]] > 0) & (q.T[[0, 3, 5]] < F(7e4))).all(0) & (r01 < 1) & (r02 < 1) & (r12 < 1)
        return np.where(ok & (det >= F(1.0 / 250.0)), F(9.1), F(np.inf))


def _separated(q, e):
    q00, h01, h02, q11, h12, q22 = (x[:, None] for x in q.T)
    e0, e1, e2 = (e[..., k] for k in range(3))
    n0, n1, n2 = q00 * e0 + h01 * e1 + h02 * e2, h01 * e0 + q11 * e1 + h12 * e2, h02 * e0 + h12 * e1 + q22 * e2
    m = n0 * e0 + n1 * e1 + n2 * e2
    t = F(0.99) * m - F(1.515) * (np.abs(n0) + np.abs(n1) + np.abs(n2))
    with np.errstate(all="ignore"):
        return (t > 0) & (t * t > _threshold(q)[:, None] * m)


@pytest.mark.parametrize("spread", [0.2, 1.0, 2.0, 3.5])
def test_no_separated_block_holds_an_included_voxel(spread):
    rng = np.random.default_rng(int(10 * spread))
    n, blocks = 3000, 160
    sig = np.exp(rng.normal(np.log(1.5), spread, (n, 3)))
    quat = rng.normal(size=(n, 4))
    quat[: n // 4, 1:] *= 1e-3  # nearly axis-aligned
    w, x, y, z = (quat / np.linalg.norm(quat, axis=1, keepdims=True)).T
    rot = np.stack([1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w), 2 * (x * y + z * w),
                    1 - 2 * (x * x + z * z), 2 * (y * z - x * w), 2 * (x * z - y * w), 2 * (y * z + x * w),
                    1 - 2 * (x * x + y * y)], -1).reshape(n, 3, 3)
    t = rot / sig[:, None, :]
    Q = np.einsum("nij,nkj->nik", t, t)
    q = Q[:, [0, 0, 0, 1, 1, 2], [0, 1, 2, 1, 2, 2]].astype(F)
    # block centres on a shell around the inclusion set's surface, where the rule decides
    u = rng.normal(size=(n, blocks, 3))
    u /= np.linalg.norm(u, axis=-1, keepdims=True)
    surf = 3.0 * np.einsum("nij,nbj->nbi", rot * sig[:, None, :], u)
    e = (surf + rng.uniform(-4, 4, (n, blocks, 3))).astype(F)
    sep = _separated(q, e)
    off = np.stack(np.meshgrid(*[np.arange(4) - 1.5] * 3, indexing="ij"), -1).reshape(-1, 3)
    # m of every voxel of every block with the stored coefficients, in 64 bits
    qs = q.astype(np.float64)
    Qs = qs[:, [0, 1, 2, 1, 3, 4, 2, 4, 5]].reshape(n, 3, 3)
    lowest = np.full((n, blocks), np.inf)
    for o in off:
        v = e.astype(np.float64) + o
        lowest = np.minimum(lowest, np.einsum("nbi,nij,nbj->nb", v, Qs, v))
    assert not (sep & (lowest <= 9 * (1 + 8.3e-4))).any()
    assert sep.any()
