"""The FP64 form's contractions over grid points where their operands are graded against one another: steep functions,
largest where the integration weights are smallest, beside diffuse ones.

Bound, element by element.  A row is fixed point on its largest value after each point's power of two (half the
exponent of the point's largest coefficient, relative to the spin's largest; of the two spins' the larger), 61 bits, and the products left out are below 2^-58 of the product of the
rows' powers of two.  Those are at most twice the largest phi 2^t and 2^5 times the largest term of Q 2^-t (three
octaves for the sum of five terms, a quarter for the approximate product, one for the mantissa), so 2^-52 of the
product of these maxima for each point.  Without the octaves the maxima are those of phi and Q themselves, thousands
of times the bound for the steepest pair.  What remains are FP64 roundings: of the five terms, of at most 320 partial
sums, and the CPU's N."""
import numpy as np
import pytest
import torch

from test_gpu_fx import E, U  # noqa: F401

pytestmark = pytest.mark.gpu

ALPHAS = np.array([1e10, 1e8, 1e6, 6665.0, 30.0, 1.0, 0.15])


def _octaves(c):
    """2^t of the points or AOs: t half the difference of the high words of the largest |c| there and of the spin's
    largest, in octaves (floor), the larger of the spins'; c (spin, k, points); 0 where there is none."""
    hi = (np.ascontiguousarray(np.abs(c).max(1)).view(np.int64) >> 32).astype(np.int64)
    t = (hi - hi.max(1, keepdims=True)) >> 21
    t = np.where(hi > 0, t, -1200).max(0)
    return np.where(t > -1200, 2.0 ** np.maximum(t, -1023), 0.0)


def _tables(N, seed):
    """s functions on one centre, on a logarithmic radial grid with its weights."""
    g = np.random.default_rng(seed)
    r = np.exp(np.linspace(np.log(1e-7), np.log(12.0), N))
    u = g.standard_normal((N, 3))
    x = r[:, None] * u / np.linalg.norm(u, axis=1, keepdims=True)
    w = 4 * np.pi * r ** 3 * np.log(12.0 / 1e-7) / N
    phi = (2 * ALPHAS / np.pi) ** 0.75 * np.exp(-ALPHAS * r[:, None] ** 2)
    g1 = -2 * ALPHAS[None, :, None] * x[:, None] * phi[..., None]
    g2 = (4 * ALPHAS[None, :, None] ** 2 * x[:, None] ** 2 - 2 * ALPHAS[None, :, None]) * phi[..., None]
    v = (50 * np.exp(-16 * r) + 0.5 * np.exp(-2 * r)) ** (1 / 3)
    return phi, g1, g2, x, w, v


@pytest.mark.parametrize("terms", ["rho", "gradient", "all"])
def test_vxc(E, terms):  # noqa: F811
    N = 300
    phi, g1, g2, x, w, v = _tables(N, 1)
    n = len(ALPHAS)
    pot = np.zeros((2, 6, N))
    pot[:, 0] = -w * v
    if terms != "rho":
        pot[:, 1:4] = 0.1 * (w * v)[None, None] * x.T[None]
    if terms == "all":
        pot[:, 4], pot[:, 5] = 1e-3 * w * v, 0.02 * w * v
    pot[1] *= 0.7
    r = E.Resident.from_tables(phi, g1, g2, np.ones(N), "fp64", "cuda:0")
    got = r.vxc_from_potentials(pot).cpu().numpy()
    assert r.status() == 0
    lap = g2.sum(-1)
    t0, t1 = _octaves(pot[:, :5])[:, None], _octaves(pot[:, 5:])[:, None]
    for s in range(2):
        c = pot[s][..., None]
        each = [c[0] * phi, *(c[1 + j] * g1[..., j] for j in range(3)), c[4] * lap]
        ref, size = phi.T @ sum(each), np.abs(phi).T @ sum(np.abs(t) for t in each)
        lost = np.abs(phi * t0).max(0)[:, None] * np.max([np.abs(t / t0) for t in each], (0, 1))[None]
        kin = np.zeros((n, n))
        for j in range(3):
            ref += g1[..., j].T @ (c[5] * g1[..., j])
            size += np.abs(g1[..., j]).T @ np.abs(c[5] * g1[..., j])
        if pot[s, 5].any():
            kin = np.abs(g1 * t1[..., None]).max((0, 2))[:, None] * np.abs(c[5][..., None] * g1 / t1[..., None]).max((0, 2))
        bound = (320 + N + 10) * U * size + N * 2.0 ** -52 * (lost + 3 * np.maximum(kin, kin.T))
        assert np.all(np.abs(got[s] - ref) <= bound), np.max(np.abs(got[s] - ref) / bound)


def test_exact_exchange_fock(E):  # noqa: F811
    """F = ao^T B with B = -1/2 sum_w g chi: the octaves are those of each spin's g, and both rows' powers of two are at
    most twice their largest values, 2^-56 of whose product is lost for each point."""
    N, n = 300, len(ALPHAS)
    phi, _, _, _, w, v = _tables(N, 2)
    chi = phi[:, None, None] * np.random.default_rng(3).uniform(0.5, 1.0, (N, 2, 2, 1))
    g = -(w * v)[None, None] * np.array([1.0, 0.6])[:, None, None] * np.array([1.0, 0.7])[None, :, None]
    c = lambda x: torch.as_tensor(x, device="cuda")  # noqa: E731
    got = E.hf_fock(c(phi), c(chi), c(g)).cpu().numpy()
    for s in range(2):
        t = 2.0 ** ((np.frexp(np.abs(g[:, s]).max(0))[1] - 1) // 2)[:, None]
        B = -0.5 * sum(g[o, s][:, None] * chi[:, o, s] for o in range(2))
        size = np.abs(phi).T @ np.abs(B)
        bound = (N + 200) * U * size + N * 2.0 ** -56 * np.abs(phi * t).max(0)[:, None] * np.abs(B / t).max(0)
        assert np.all(np.abs(got[s] - phi.T @ B) <= bound), np.max(np.abs(got[s] - phi.T @ B) / bound)


@pytest.mark.parametrize("faint", [0.0, 1e-9, 1.0])
def test_density(E, faint):  # noqa: F811
    """Features of density matrices that hold little of the two steepest functions.  phi_a is taken times 2^t, D_ab
    times 2^-t, t from D's largest entry in row or column a as above: X is off by 2^-56 of the product of these
    rows' largest values for each of n products (2^-55 where D + D^T is contracted), tau by such sums over d_j phi."""
    N = 300
    phi, g1, g2, *_ = _tables(N, 4)
    n = len(ALPHAS)
    scale = np.where(np.arange(n) < 2, faint, 1.0)
    D = []
    for s in range(2):
        q = np.linalg.qr(np.random.default_rng(s).standard_normal((n, n)))[0][:, :3] * scale[:, None]
        D.append(q @ q.T)
    D = np.array(D)
    r = E.Resident.from_tables(phi, g1, g2, np.ones(N), "fp64", "cuda:0")
    out = {k: v.cpu().numpy() for k, v in r.density(D).items()}
    assert r.status() == 0
    t = _octaves(np.concatenate([D, D.transpose(0, 2, 1)], 1))
    lap, k = g2.sum(-1), 2 * n + 20
    for s in range(2):
        X, aX = phi @ D[s], np.abs(phi) @ np.abs(D[s])
        scaled = np.divide(np.abs(D[s]), t[:, None], out=np.zeros((n, n)), where=t[:, None] > 0).max(0)
        lost = lambda a, eps: n * 2.0 ** eps * (np.abs(a) * t).max(1)[:, None] * scaled  # noqa: E731

        def check(got, ref, size, extra):
            bound = k * U * size + extra + 1e-290
            assert np.all(np.abs(got - ref) <= bound), np.max(np.abs(got - ref) / bound)

        check(out["rho"][:, s], (X * phi).sum(1), (aX * np.abs(phi)).sum(1), (lost(phi, -56) * np.abs(phi)).sum(1))
        kin, akin, klost = np.zeros(N), np.zeros(N), np.zeros(N)
        for j in range(3):
            g = g1[..., j]
            check(out["grad_rho"][:, s, j], 2 * (X * g).sum(1), 2 * (aX * np.abs(g)).sum(1),
                  2 * (lost(phi, -56) * np.abs(g)).sum(1))
            kin += ((g @ D[s]) * g).sum(1)
            akin += ((np.abs(g) @ np.abs(D[s])) * np.abs(g)).sum(1)
            klost += (lost(g, -55) * np.abs(g)).sum(1)
        check(out["tau"][:, s], kin / 2, akin / 2, klost / 2)
        check(out["lapl"][:, s], 2 * kin + 2 * (X * lap).sum(1), 2 * akin + 2 * (aX * np.abs(lap)).sum(1),
              2 * klost + 2 * (lost(phi, -56) * np.abs(lap)).sum(1))


def test_exact_exchange_energy(E):  # noqa: F811
    """ehf = -1/2 sum_b chi_b X_b with X = ao D as in the density, D holding nothing of the four steepest functions."""
    N, n = 300, len(ALPHAS)
    phi, *_ = _tables(N, 5)
    chi = np.random.default_rng(6).standard_normal((N, 1, 2, n))
    D = np.random.default_rng(7).standard_normal((2, n, n))
    D[:, :4] = D[:, :, :4] = 0.0
    got = E.hf_energy_density(*(torch.as_tensor(x, device="cuda") for x in (phi, D, chi))).cpu().numpy()
    for s in range(2):
        t = _octaves(np.concatenate([D[s], D[s].T])[None])
        c = np.abs(chi[:, 0, s])
        scaled = (np.abs(D[s, 4:]) / t[4:, None]).max(0)
        bound = (2 * n + 20) * U * (np.abs(phi) @ np.abs(D[s]) * c).sum(1)
        bound += n * 2.0 ** -56 * (np.abs(phi) * t).max(1) * (scaled * c).sum(1)
        assert np.all(np.abs(got[0, s] + 0.5 * (chi[:, 0, s] * (phi @ D[s])).sum(1)) <= bound)


@pytest.mark.parametrize("spin", [0, 1])
def test_spins_of_different_size(E, spin):  # noqa: F811
    """The spins share the digits of phi: an entry of one spin's D or potentials that is larger by 2^440 takes nothing
    from the other spin's results."""
    n, N = 40, 300
    g = np.random.default_rng(12)
    ao, g1, g2 = (g.standard_normal((N, n) + s) for s in ((), (3,), (3,)))
    D, pot = g.standard_normal((2, n, n)), g.standard_normal((2, 6, N))
    D[spin, 3, 7], pot[spin, :, 11] = 2.0 ** 440, 2.0 ** 440
    r = E.Resident.from_tables(ao, g1, g2, np.ones(N), "fp64", "cuda:0")
    rho, v = r.density(D)["rho"].cpu().numpy(), r.vxc_from_potentials(pot).cpu().numpy()
    s, lap = 1 - spin, g2.sum(-1)
    size = ((np.abs(ao) @ np.abs(D[s])) * np.abs(ao)).sum(1)
    assert np.all(np.abs(rho[:, s] - ((ao @ D[s]) * ao).sum(1)) <= 4 * n * U * size)
    c = pot[s][..., None]
    each = [c[0] * ao, *(c[1 + j] * g1[..., j] for j in range(3)), c[4] * lap]
    ref, size = ao.T @ sum(each), np.abs(ao).T @ sum(np.abs(t) for t in each)
    for j in range(3):
        ref += g1[..., j].T @ (c[5] * g1[..., j])
        size += np.abs(g1[..., j]).T @ np.abs(c[5] * g1[..., j])
    assert np.all(np.abs(v[s] - ref) <= (N + 400) * U * size)  # 2^-52 of maxima of a few units is well inside
