"""The separating-plane cull for flat and needle-shaped Gaussians (``plane_by_k`` in gsv_common.cuh): the
rule restated in float32 with its threshold and factor by the anisotropy K.  No block it rules out may
hold a voxel that the row form of the quadratic could include (m <= 9 (1 + 3.3e-6 K)), up to the K where
it is switched off, for coefficients up to its limit, and it does rule blocks out."""
import numpy as np
import pytest

F = np.float32


def _rule(q):
    """(threshold, factor) of each Gaussian: K in 64 bits from the stored coefficients."""
    q00, q01, q02, q11, q12, q22 = q.astype(np.float64).T
    c00, c11, c22 = q11 * q22 - q12 * q12, q00 * q22 - q02 * q02, q00 * q11 - q01 * q01
    det = q00 * c00 + q01 * (q02 * q12 - q01 * q22) + q02 * (q01 * q12 - q02 * q11)
    ok = (q00 > 0) & (c22 > 0) & (det > 0) & (c00 > 0) & (c11 > 0)
    with np.errstate(all="ignore"):
        k = np.where(ok, np.max([q00 * c00, q11 * c11, q22 * c22], axis=0) / det, np.inf)
    top = np.max([q00, q11, q22], axis=0)
    thr = np.where(k <= 1000, F(9.35), F(11.2))
    thr = np.where((top < 1.7e4) & (k <= 1e4), thr, np.inf)
    thr = np.where((k <= 250) & (top < 7e4), F(9.1), thr).astype(F)
    return k, thr, np.where(thr < 10, F(0.99), F(0.9)).astype(F)


def _separated(q, e, thr, factor):
    q00, h01, h02, q11, h12, q22 = (x[:, None] for x in q.T)
    e0, e1, e2 = (e[..., k] for k in range(3))
    n0, n1, n2 = q00 * e0 + h01 * e1 + h02 * e2, h01 * e0 + q11 * e1 + h12 * e2, h02 * e0 + h12 * e1 + q22 * e2
    m = n0 * e0 + n1 * e1 + n2 * e2
    t = factor[:, None] * m - F(1.515) * (np.abs(n0) + np.abs(n1) + np.abs(n2))
    with np.errstate(all="ignore"):
        return (t > 0) & (t * t > thr[:, None] * m)


@pytest.mark.parametrize("ratio", [10, 33, 70, 150])
@pytest.mark.parametrize("thin", [0.008, 0.05, 0.4])
@pytest.mark.parametrize("form", ["pancake", "needle"])
def test_no_separated_block_holds_an_included_voxel(form, thin, ratio):
    rng = np.random.default_rng(ratio)
    n, blocks = 1500, 200
    sig = np.where(np.array([1, 0, 0]) > 0, thin, thin * ratio) if form == "pancake" else np.array([thin, thin, thin * ratio])
    sig = sig * np.exp(rng.normal(0, 0.2, (n, 3)))
    quat = rng.normal(size=(n, 4))
    w, x, y, z = (quat / np.linalg.norm(quat, axis=1, keepdims=True)).T
    rot = np.stack([1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w), 2 * (x * y + z * w),
                    1 - 2 * (x * x + z * z), 2 * (y * z - x * w), 2 * (x * z - y * w), 2 * (y * z + x * w),
                    1 - 2 * (x * x + y * y)], -1).reshape(n, 3, 3)
    t = rot / sig[:, None, :]
    Q = np.einsum("nij,nkj->nik", t, t)
    q = Q[:, [0, 0, 0, 1, 1, 2], [0, 1, 2, 1, 2, 2]].astype(F)
    k, thr, factor = _rule(q)
    # block centres around the inclusion set's surface, and some farther off
    u = rng.normal(size=(n, blocks, 3))
    u /= np.linalg.norm(u, axis=-1, keepdims=True)
    e = (3.0 * np.einsum("nij,nbj->nbi", rot * sig[:, None, :], u) + rng.uniform(-4, 4, (n, blocks, 3))).astype(F)
    sep = _separated(q, e, thr, factor)
    off = np.stack(np.meshgrid(*[np.arange(4) - 1.5] * 3, indexing="ij"), -1).reshape(-1, 3)
    qs = q.astype(np.float64)
    Qs = qs[:, [0, 1, 2, 1, 3, 4, 2, 4, 5]].reshape(n, 3, 3)
    lowest = np.full((n, blocks), np.inf)
    for o in off:
        v = e.astype(np.float64) + o
        lowest = np.minimum(lowest, np.einsum("nbi,nij,nbj->nb", v, Qs, v))
    limit = 9 * (1 + 3.3e-6 * np.minimum(k, 1e4))
    assert not (sep & (lowest <= limit[:, None])).any()
    on = np.isfinite(thr)
    if on.any():
        assert sep[on].any()
    assert not sep[~on].any()
