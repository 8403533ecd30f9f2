"""Direct sums and energies at the remainders of their tiles, warps and clusters, against FP64 on the host.

Tolerances: an FP32 term carries a reciprocal root good to about 2^-22 (cubed) and some ten roundings, an
FP64 term some ten roundings of 2^-53, and sums of a few thousand terms add far less than that again;
bounds are relative to the sum of the terms' magnitudes.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def reference(bodies, targets, eps):
    d = bodies[None, :, :3].astype(np.float64) - targets[:, None, :3].astype(np.float64)
    d2 = (d * d).sum(-1)
    w = np.zeros_like(d2)
    np.divide(bodies[None, :, 3].astype(np.float64), (d2 + eps) ** 1.5, out=w, where=d2 > 0)
    terms = d * w[..., None]
    return terms.sum(1), np.abs(terms).sum(1)


@pytest.mark.parametrize("n,nt", [(1, 1), (2, 33), (255, 31), (256, 32), (257, 300), (1025, 1), (4097, 513), (20011, 64), (700, 8191), (700, 8192), (700, 8257)])
@pytest.mark.parametrize("eps", [0.0, 1e-4])
def test_direct_sums(nb, n, nt, eps):
    import torch

    pm, _ = nb.scenarios.plummer(max(n, 8), seed=n + nt)
    pm = pm[:n]
    rng = np.random.default_rng(n)
    targets = np.concatenate([pm, rng.uniform(-2, 2, (nt, 4)).astype(np.float32)])[-nt:] if n % 2 else pm[np.arange(nt) % n]
    eps = float(np.float32(eps))
    ref, size = reference(pm, targets, eps)
    b, t = torch.from_numpy(pm).cuda(), torch.from_numpy(np.ascontiguousarray(targets)).cuda()
    a32 = torch.zeros(nt, 4, device="cuda")
    a64 = torch.zeros(nt, 3, device="cuda", dtype=torch.float64)
    torch.cuda.synchronize()
    with nb.NaiveSolver(None, nb.Gravity(1.0, eps)) as s:
        s.direct_device(n, b.data_ptr(), nt, t.data_ptr(), a32.data_ptr(), 32)
        s.direct_device(n, b.data_ptr(), nt, t.data_ptr(), a64.data_ptr(), 64)
        s.synchronize()
    assert (np.abs(a32.cpu().numpy()[:, :3] - ref) <= 4e-6 * size).all()
    assert (np.abs(a64.cpu().numpy() - ref) <= 2e-14 * size).all()


def test_wide_direct_sums(nb):
    import torch

    pm, _ = nb.scenarios.plummer(300, seed=3)
    nt = 300_037  # one warp in eight per tile; the wide forms: test_wide_lines
    t = torch.from_numpy(pm[np.arange(nt) % 300]).cuda()
    b = torch.from_numpy(pm).cuda()
    a32 = torch.zeros(nt, 4, device="cuda")
    a64 = torch.zeros(nt, 3, device="cuda", dtype=torch.float64)
    torch.cuda.synchronize()
    ref, size = reference(pm, pm, float(np.float32(1e-4)))
    with nb.NaiveSolver(None, nb.Gravity(1.0, 1e-4)) as s:
        s.direct_device(300, b.data_ptr(), nt, t.data_ptr(), a32.data_ptr(), 32)
        s.direct_device(300, b.data_ptr(), nt, t.data_ptr(), a64.data_ptr(), 64)
        s.synchronize()
    at = np.arange(nt) % 300
    assert (np.abs(a32.cpu().numpy()[:, :3] - ref[at]) <= 4e-6 * size[at]).all()
    assert (np.abs(a64.cpu().numpy() - ref[at]) <= 2e-14 * size[at]).all()


@pytest.mark.parametrize("n,nt", [(1, 100_000), (128, 100_003), (128, 99_999), (129, 300_000), (200, 700_001)])
def test_wide_lines(nb, n, nt):
    """Both sides of the lines of the wide form, by targets and by sources."""
    import torch

    pm, _ = nb.scenarios.plummer(max(n, 8), seed=n)
    pm = pm[:n]
    own = np.concatenate([pm, np.float32([[0.5, -0.25, 0.125, 0.0]])])
    at = np.arange(nt) % len(own)
    b, t = torch.from_numpy(pm).cuda(), torch.from_numpy(own[at]).cuda()
    a32 = torch.zeros(nt, 4, device="cuda")
    a64 = torch.zeros(nt, 3, device="cuda", dtype=torch.float64)
    torch.cuda.synchronize()
    ref, size = reference(pm, own, float(np.float32(1e-4)))
    with nb.NaiveSolver(None, nb.Gravity(1.0, 1e-4)) as s:
        s.direct_device(n, b.data_ptr(), nt, t.data_ptr(), a32.data_ptr(), 32)
        s.direct_device(n, b.data_ptr(), nt, t.data_ptr(), a64.data_ptr(), 64)
        s.synchronize()
    assert (np.abs(a32.cpu().numpy()[:, :3] - ref[at]) <= 4e-6 * size[at]).all()
    assert (np.abs(a64.cpu().numpy() - ref[at]) <= 2e-14 * size[at]).all()


@pytest.mark.parametrize("n", [1, 2, 255, 256, 257, 512, 513, 1024, 1025, 5000])
@pytest.mark.parametrize("eps", [0.0, 1e-4])
def test_energy(nb, n, eps):
    pm, vel = nb.scenarios.plummer(max(n, 8), seed=n)
    pm, vel = pm[:n].copy(), vel[:n]
    if n > 300:
        pm[300, :3] = pm[10, :3]  # coincident bodies in different tiles
        pm[301, :3] = pm[300, :3]
    eps = float(np.float32(eps))
    p = pm.astype(np.float64)
    u = 0.0
    for i in range(n):
        d2 = ((p[:, :3] - p[i, :3]) ** 2).sum(1)
        on = d2 > 0
        u += p[i, 3] * (p[on, 3] / np.sqrt(d2[on] + eps)).sum()
    k = 0.5 * (p[:, 3] * (vel[:, :3].astype(np.float64) ** 2).sum(1)).sum()
    with nb.NaiveSolver(pm, nb.Gravity(1.0, eps), vel) as s:
        kinetic, potential = s.energy()
    assert abs(kinetic - k) <= 1e-14 * k
    assert abs(potential + 0.5 * u) <= 1e-14 * max(u, 1e-300)


@pytest.mark.parametrize("precision", [32, 64])
def test_infinite_distances_add_zero(nb, precision):
    """A source at infinity along one axis leaves the other axes' sums alone, a target there has none along
    them, and infinite softening leaves no sum at all."""
    import torch

    pm, vel = nb.scenarios.plummer(300, seed=9)
    far = np.array([[np.inf, 0.25, -0.5, 1.0]], np.float32)

    def sums(bodies, eps, targets=pm[:40]):
        b, t = torch.from_numpy(bodies).cuda(), torch.from_numpy(targets.copy()).cuda()
        acc = torch.zeros(len(targets), 4 if precision == 32 else 3, device="cuda",
                          dtype=torch.float32 if precision == 32 else torch.float64)
        torch.cuda.synchronize()
        with nb.NaiveSolver(None, nb.Gravity(1.0, eps)) as s:
            s.direct_device(len(bodies), b.data_ptr(), len(targets), t.data_ptr(), acc.data_ptr(), precision)
            s.synchronize()
        return acc.cpu().numpy()[:, :3]

    eps = float(np.float32(1e-4))
    ref, size = reference(pm, pm[:40], eps)
    got = sums(np.concatenate([pm[:100], far, pm[100:]]), eps)
    assert np.isnan(got[:, 0]).all()
    assert (np.abs(got[:, 1:] - ref[:, 1:]) <= (4e-6 if precision == 32 else 2e-14) * size[:, 1:]).all()
    got = sums(pm, eps, far)
    assert np.isnan(got[0, 0]) and (got[0, 1:] == 0).all()
    assert (sums(pm, np.inf) == 0).all()
    with nb.NaiveSolver(pm, nb.Gravity(1.0, np.inf), vel) as s:
        assert s.energy()[1] == 0.0


# One term each, so that the reciprocal root's error shows. With u = 2^-53, differences to a body at the origin
# exact and G = 1: |r|^2 + eps carries 4 u, its root 2 u and u of its own; the force's factor takes three times
# that, three products and the product with the difference, 13 u in all (14 u allowed); the potential the root, two
# products and one sum, 6 u (7 u allowed). The reference is in extended precision.
ULP = np.longdouble(2.0) ** -53


@pytest.mark.parametrize("eps", [0.0, 1e-4])
def test_fp64_force_term(nb, eps):
    import torch

    rng = np.random.default_rng(11)
    nt = 20000
    d = rng.standard_normal((nt, 3))
    t = np.zeros((nt, 4), np.float32)
    t[:, :3] = d / np.linalg.norm(d, axis=1)[:, None] * 10.0 ** rng.uniform(-6, 6, (nt, 1))
    source = np.array([[0.0, 0.0, 0.0, 0.37]], np.float32)
    eps = np.float32(eps)
    b, tt = torch.from_numpy(source).cuda(), torch.from_numpy(t).cuda()
    acc = torch.zeros(nt, 3, device="cuda", dtype=torch.float64)
    torch.cuda.synchronize()
    with nb.NaiveSolver(None, nb.Gravity(1.0, float(eps))) as s:
        s.direct_device(1, b.data_ptr(), nt, tt.data_ptr(), acc.data_ptr(), 64)
        s.synchronize()
    x = t[:, :3].astype(np.longdouble)
    r2 = (x * x).sum(1) + np.longdouble(eps)
    ref = -x * (np.longdouble(source[0, 3]) / (r2 * np.sqrt(r2)))[:, None]
    assert (np.abs(acc.cpu().numpy().astype(np.longdouble) - ref) <= 14 * ULP * np.abs(ref)).all()


@pytest.mark.parametrize("eps", [0.0, 1e-4])
def test_fp64_potential_term(nb, eps):
    rng = np.random.default_rng(12)
    eps = np.float32(eps)
    with nb.NaiveSolver(None, nb.Gravity(1.0, float(eps))) as s:
        for k in range(60):
            pm = np.zeros((2, 4), np.float32)
            pm[1, :3] = rng.standard_normal(3) * 10.0 ** rng.uniform(-6, 6)
            pm[:, 3] = rng.uniform(0.1, 2.0, 2)
            s.set_bodies(pm)
            x = pm.astype(np.longdouble)
            ref = -x[0, 3] * x[1, 3] / np.sqrt((x[1, :3] ** 2).sum() + np.longdouble(eps))
            assert abs(np.longdouble(s.energy()[1]) - ref) <= 7 * ULP * abs(ref)
