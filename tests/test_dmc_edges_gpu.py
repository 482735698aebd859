"""SparseDiffDMC where its passes change form: a handful of cubes with random
signs (ambiguous cases checked against neighbours that are there or not, edges
shared by one to four cubes), and the adjoint of L_dev with and without alpha
weights (with alpha the weighted and the plain crossing differ)."""

import numpy as np
import pytest
import torch

from atom3d_b200 import SparseDiffDMC, synthetic

pytestmark = pytest.mark.gpu

TOL = 1e-6 * 2 * np.sqrt(3)


def _cubes(n, res, seed):
    g = np.random.default_rng(seed)
    flat = np.sort(g.choice(res ** 3, size=n, replace=False))
    vox = np.stack([flat // res ** 2, (flat // res) % res, flat % res], 1)
    corner = np.stack([[c & 1, (c >> 1) & 1, (c >> 2) & 1] for c in range(8)])
    p = vox[:, None] + corner[None]
    q = res + 1
    ids, inv = np.unique((p[..., 0] * q + p[..., 1]) * q + p[..., 2], return_inverse=True)
    sdf = g.uniform(0.1, 1.0, ids.size) * np.where(g.random(ids.size) < 0.5, -1, 1)
    return vox.astype(np.int64), sdf.astype(np.float32), inv.reshape(-1, 8).astype(np.int64)


@pytest.mark.parametrize("n,res", [(1, 2), (2, 2), (8, 2), (31, 4), (33, 4), (64, 4), (300, 7), (1331, 11)])
def test_few_cubes_of_random_signs(n, res):
    from oracle import dmc_oracle as D

    vox, sdf, cidx = _cubes(n, res, 100 + n)
    o = SparseDiffDMC(device="cuda")(*(torch.from_numpy(a).cuda() for a in (vox, sdf, cidx)), res)
    r = D.forward(vox, sdf, cidx, res)
    assert np.array_equal(o.faces.cpu().numpy(), r["faces"])
    for k in ("vertices", "L_dev", "p_alpha", "n_alpha"):
        a = getattr(o, k).cpu().numpy()
        assert a.shape == r[k].shape, k
        assert a.size == 0 or np.abs(a - r[k]).max() <= TOL, k


@pytest.mark.parametrize("weights", [False, True])
def test_ldev_adjoint_vs_fp64_differences(weights):
    from oracle import dmc_oracle as D

    vox, sdf, cidx, _ = synthetic.dmc_spheres(res=20, seed=4, n_spheres=3, noise=0.0)
    rng = np.random.default_rng(1)
    kw = {}
    if weights:
        kw = {"alpha": rng.normal(0, 0.3, (vox.shape[0], 8)), "beta": rng.normal(0, 0.3, (vox.shape[0], 12))}
    kw = {k: v.astype(np.float32) for k, v in kw.items()}
    s = torch.from_numpy(sdf.numpy()).cuda().requires_grad_(True)
    o = SparseDiffDMC(device="cuda")(vox.cuda(), s, cidx.cuda(), 20, **{k: torch.from_numpy(v).cuda()
                                                                       for k, v in kw.items()})
    w = rng.normal(size=o.L_dev.shape[0])
    wv = rng.normal(size=tuple(o.vertices.shape))
    wt, wvt = (torch.from_numpy(a).float().cuda() for a in (w, wv))
    ((o.L_dev * wt).sum() * 20 + (o.vertices * wvt).sum()).backward()
    g = s.grad.cpu().double().numpy()

    def loss(x):
        r = D.forward(vox.numpy(), x, cidx.numpy(), 20, dtype=np.float64, **kw)
        return 20 * (r["L_dev"] * w.astype(np.float32)).sum() + (r["vertices"] * wv.astype(np.float32)).sum()

    x0 = sdf.double().numpy()
    f0 = loss(x0)
    # central differences in FP64; L_dev has kinks (|distance - mean|), at
    # which the one-sided differences disagree: those samples say nothing.
    # The FP32 adjoint errs by some 1e-6 of sums of terms up to the largest
    # gradient; the differences by h * curvature, below 1e-3 of it at h = 1e-7.
    h, tol = 1e-7, 2e-3 * np.abs(g).max()
    used = 0
    for i in rng.choice(np.nonzero(g)[0], size=30, replace=False):
        d = np.zeros_like(x0)
        d[i] = h
        up, down = (loss(x0 + d) - f0) / h, (f0 - loss(x0 - d)) / h
        if abs(up - down) > tol:
            continue
        used += 1
        assert abs(g[i] - 0.5 * (up + down)) <= tol, (i, g[i], up, down)
    assert used >= 15
