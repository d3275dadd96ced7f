"""mcl_measure_extras on lattices larger than one pass of its grid (each block strides over the sites), against the
formulas of src/parameter_order.cpp:129-245 in vectorised FP64."""
import numpy as np
import pytest

from helpers import M

pytestmark = pytest.mark.gpu


def directors(shape, seed):
    nx, ny, nz = shape
    z, y, x = np.meshgrid(np.arange(nz), np.arange(ny), np.arange(nx), indexing="ij")
    n = np.random.default_rng(seed).normal(size=(nz, ny, nx, 3)) * 0.4
    n += np.stack([0.5 * np.sin(2 * np.pi * x / nx), 0.4 * np.cos(2 * np.pi * z / nz), 1.0 + 0 * y], -1)
    return (n / np.linalg.norm(n, axis=-1, keepdims=True)).astype(np.float32)


def reference(n32, periodic, director):
    n = n32.astype(np.float64)
    nz, ny, nx = n.shape[:3]
    splay, bonds, div = np.zeros(3), 0.0, np.zeros(n.shape[:3])
    for a in range(3):
        axis, total, count = 2 - a, np.zeros(n.shape[:3]), np.zeros(n.shape[:3])
        for s in (1, -1):
            m, w = np.roll(n, -s, axis), np.ones(n.shape[:3])
            if not periodic[a]:
                edge = [slice(None)] * 3
                edge[axis] = -1 if s > 0 else 0
                w[tuple(edge)] = 0
            ra, rb, ab = s * n[..., a], s * m[..., a], (n * m).sum(-1)
            term = m * rb[..., None] - n * ra[..., None] + n * (ab * rb)[..., None] - m * (ab * ra)[..., None]
            splay += 0.5 * (w[..., None] * term).sum((0, 1, 2))
            bonds += w.sum()
            total += w * s * (m[..., a] - n[..., a])
            count += w
        div += total / np.maximum(count, 1)
    z, y, x = np.meshgrid(np.arange(nz) - nz // 2, np.arange(ny) - ny // 2, np.arange(nx) - nx // 2, indexing="ij")
    out = {"P": abs((n.sum((0, 1, 2)) * director).sum()) / (nx * ny * nz),
           "dtheta": 1.5 * np.linalg.norm(splay) / bonds, "divn": div.mean()}
    for name, rz in (("sph", z), ("cyl", 0 * z)):
        r = np.stack([x, y, rz], -1).astype(float)
        length = np.linalg.norm(r, axis=-1)
        c = ((n * r).sum(-1) / np.maximum(length, 0.5))[length >= 0.5]
        out["Sr_" + name], out["Pr_" + name] = (1.5 * c * c - 0.5).mean(), c.mean()
    return out


@pytest.mark.parametrize("shape,periodic", [((97, 61, 53), (0, 0, 0)), ((128, 64, 40), (1, 1, 1)),
                                            ((98, 75, 44), (1, 0, 1))])
def test_extras_on_more_sites_than_the_grid_has_threads(shape, periodic):
    n = directors(shape, 3)
    assert n.size // 3 > 148 * 8 * 256
    e = M.Engine(M.Model("pear"), [M.Replica(*shape, "bulk", periodic, T=0.5, seed=3)])
    e.upload(0, n.reshape(-1))
    d = np.array([0.2, -0.1, 0.97])
    got, ref = e.measure_extras(0, d), reference(n, periodic, d.astype(np.float32).astype(np.float64))
    e.close()
    for key in ref:  # FP32 site terms: the tolerance of the small lattices' test
        assert abs(got[key] - ref[key]) <= 2e-6 + 2e-6 * abs(ref[key]), (key, got[key], ref[key])
