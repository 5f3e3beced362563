"""The FP64 form's contractions on digit products (csrc/fx_*.cu) at the edges of their tiles, against torch float64
sums on the CPU, and their way to the plain kernels when an operand is not finite.

Bounds, element by element, from the arithmetic.  Digits keep 61 bits of a row's largest value and the products that
are left out are below 2^-60 of the largest product, so each product of two rows is off by less than 2^-57 of the
product of their largest values.  What remains are FP64 roundings of 2^-53: one of each X, the n / 8 + 11 additions of
a feature; for V the additions of at most 320 partial sums.  The CPU sums have their own n (or N) roundings.
"""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

U = 2.0 ** -53


@pytest.fixture(scope="module")
def E(built_lib):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from graddft_gb300 import engine

    return engine


def _tables(n, N, seed):
    """Tables with rows and columns of very different sizes (10^-20 .. 10^2), a non-symmetric D."""
    g = np.random.default_rng(seed)
    scale = 10.0 ** g.uniform(-3, 2, n)[None, :] * 10.0 ** g.uniform(-17, 0, N)[:, None]
    ao, g1, g2 = (g.standard_normal((N, n) + s) * (scale if not s else scale[..., None]) for s in ((), (3,), (3,)))
    ao[g.integers(0, N, max(1, N // 7))] = 0.0
    return ao, g1, g2, g.standard_normal((2, n, n)), g.standard_normal((2, 6, N)) * 10.0 ** g.uniform(-6, 3, N)


def _dot_bound(x, y, k):
    """(k roundings of sum_c |x| |y|) + what the digits leave out, both times the row maxima."""
    return k * U * (np.abs(x) * np.abs(y)).sum(-1)


def _resident(E, ao, g1, g2):
    return E.Resident.from_tables(ao, g1, g2, np.ones(ao.shape[0]), "fp64", "cuda:0")


SIZES = [(1, 1), (7, 127), (31, 128), (33, 129), (63, 640), (64, 65), (65, 257), (128, 300), (129, 1000), (193, 500),
         (130, 30001), (7, 300001)]  # the last crosses the slabs of both contractions


@pytest.mark.parametrize("n,N", SIZES)
def test_density_features(E, n, N):
    ao, g1, g2, D, _ = _tables(n, N, 100 * n + N)
    r = _resident(E, ao, g1, g2)
    out = {k: v.cpu().numpy() for k, v in r.density(D).items()}
    r.status()
    only = {k: v.cpu().numpy() for k, v in r.density(D, want=("rho", "grad_rho")).items() if v is not None}
    lap = g2.sum(-1)
    k = n + n / 8 + 14  # the CPU's product and ours
    for s in range(2):
        X, aX = ao @ D[s], np.abs(ao) @ np.abs(D[s])
        # What digits may lose in X: the row's and the column's largest values, n products.
        lost = 2.0 ** -57 * n * np.abs(ao).max(1)[:, None] * np.abs(D[s]).max(0)[None]

        def check(got, ref, x, y, extra, what):
            bound = _dot_bound(x, y, k) + extra + 1e-300
            assert np.all(np.abs(got - ref) <= bound), (what, np.max(np.abs(got - ref) / bound))

        check(out["rho"][:, s], (X * ao).sum(1), aX, ao, (lost * np.abs(ao)).sum(1), "rho")
        np.testing.assert_array_equal(only["rho"][:, s], out["rho"][:, s])
        for j in range(3):
            check(out["grad_rho"][:, s, j] / 2, (X * g1[..., j]).sum(1), aX, g1[..., j],
                  (lost * np.abs(g1[..., j])).sum(1), "grad")
            np.testing.assert_array_equal(only["grad_rho"][:, s, j], out["grad_rho"][:, s, j])
        kin, akin, klost = np.zeros(N), np.zeros(N), np.zeros(N)
        for j in range(3):
            kin += ((g1[..., j] @ D[s]) * g1[..., j]).sum(1)
            akin += ((np.abs(g1[..., j]) @ np.abs(D[s])) * np.abs(g1[..., j])).sum(1)
            klost += (2.0 ** -56 * n * np.abs(g1[..., j]).max(1) * np.abs(D[s]).max() * np.abs(g1[..., j]).sum(1))
        kb = (k + 4) * U * akin + klost + 1e-300
        assert np.all(np.abs(out["tau"][:, s] * 2 - kin) <= kb)
        lb = 2 * kb + 2 * (_dot_bound(aX, lap, k) + (lost * np.abs(lap)).sum(1))
        assert np.all(np.abs(out["lapl"][:, s] - 2 * kin - 2 * (X * lap).sum(1)) <= lb)


@pytest.mark.parametrize("n,N", SIZES)
@pytest.mark.parametrize("kinetic", [True, False])
def test_vxc(E, n, N, kinetic):
    ao, g1, g2, _, pot = _tables(n, N, 100 * n + N + 1)
    if not kinetic:
        pot[:, 5] = 0.0
    r = _resident(E, ao, g1, g2)
    got = r.vxc_from_potentials(pot).cpu().numpy()
    r.status()
    lap = g2.sum(-1)
    for s in range(2):
        c = pot[s][..., None]
        Q = c[0] * ao + sum(c[1 + j] * g1[..., j] for j in range(3)) + c[4] * lap
        aQ = np.abs(c[0] * ao) + sum(np.abs(c[1 + j] * g1[..., j]) for j in range(3)) + np.abs(c[4] * lap)
        ref, size = ao.T @ Q, np.abs(ao).T @ aQ
        lost = np.abs(ao).max(0)[:, None] * aQ.max(0)[None]
        for j in range(3):
            K = c[5] * g1[..., j]
            ref += g1[..., j].T @ K
            size += np.abs(g1[..., j]).T @ np.abs(K)
            lost += np.abs(g1[..., j]).max(0)[:, None] * np.abs(K).max(0)[None]
        # The kinetic rows share one exponent over the three planes: 10^0.5 at most between them here.
        bound = (320 + N / 16 + 32) * U * size + N * 2.0 ** -52 * np.maximum(lost, lost.T) + 1e-300
        assert np.all(np.abs(got[s] - ref) <= bound), np.max(np.abs(got[s] - ref) / bound)


@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
def test_not_finite(E, value):
    """One bad entry: the plain kernels' (IEEE) pattern, and a following finite call is unaffected."""
    n, N = 40, 300
    ao, g1, g2, D, pot = _tables(n, N, 9)
    r = _resident(E, ao, g1, g2)
    clean, vclean = r.density(D), r.vxc_from_potentials(pot)
    bad = D.copy()
    bad[1, 3, 5] = value
    out = r.density(bad)
    assert torch.equal(torch.isfinite(out["rho"][:, 0]), torch.ones(N, dtype=torch.bool, device="cuda"))
    t = torch.as_tensor(ao)
    ref = ((t @ torch.as_tensor(bad[1])) * t).sum(1)
    assert torch.equal(torch.isfinite(out["rho"][:, 1].cpu()), torch.isfinite(ref))
    badpot = pot.copy()
    badpot[0, 0, 17] = value
    v = r.vxc_from_potentials(badpot).cpu().numpy()
    assert not np.isfinite(v[0]).all() and np.isfinite(v[1]).all()
    row = ao[17][:, None] * (value * ao[17])[None]
    assert np.array_equal(np.isnan(v[0]), np.isnan(row) | np.isnan(v[0])) and not np.isfinite(v[0][~np.isfinite(row)]).any()
    for k, x in r.density(D).items():
        assert torch.equal(x, clean[k])
    assert torch.equal(r.vxc_from_potentials(pot), vclean)


@pytest.mark.parametrize("width", [32, 64, 128, 256])
@pytest.mark.parametrize("rows", [1, 63, 127, 129, 1000])
def test_network_layers(E, width, rows):
    """The coefficient network on given inputs (fx_mat.cu's tall GEMMs, any number of rows) against torch float64.

    A layer's GEMM and its row statistics round at 2^-53 of sums of `width` terms; the sigmoid's input after three
    layers is of order one, so 1e-13 is some 500 roundings."""
    import graddft_gb300 as G
    from graddft_gb300 import synthetic
    import oracle as O

    f = G.DM21(layer_widths=(width,) * 3)
    p = synthetic.glorot_params(layer_widths=(width,) * 3, seed=width + rows)
    x = np.random.default_rng(rows).standard_normal((rows, 11)) * 10.0 ** np.random.default_rng(1).uniform(-8, 2, 11)
    tp = {"params": {k: {kk: torch.as_tensor(v) for kk, v in d.items()} for k, d in p["params"].items()}}
    got = f.apply(p, torch.as_tensor(x, device="cuda")).cpu()
    ref = O.dm21_network(tp, torch.as_tensor(x), n_layers=3)
    assert got.shape == ref.shape and torch.max(torch.abs(got - ref)) <= 1e-13


@pytest.mark.parametrize("n,N", [(1, 1), (13, 65), (64, 128), (65, 129), (130, 1003), (200, 400)])
def test_exact_exchange(E, n, N):
    """ehf and the exchange Fock term (fx_mat.cu's two GEMMs) at ragged sizes, element by element as above."""
    ao, _, _, D, pot = _tables(n, N, 7 * n + N)
    g = np.random.default_rng(n)
    chi, w = g.standard_normal((N, 2, 2, n)), pot[:, :2].transpose(1, 0, 2).copy()  # (omega, spin, grid)
    t = lambda v: torch.as_tensor(v, device="cuda")  # noqa: E731
    ehf = E.hf_energy_density(t(ao), t(D), t(chi)).cpu().numpy()
    fock = E.hf_fock(t(ao), t(chi), t(w)).cpu().numpy()
    for s in range(2):
        X, aX = ao @ D[s], np.abs(ao) @ np.abs(D[s])
        lost = 2.0 ** -57 * n * np.abs(ao).max(1)[:, None] * np.abs(D[s]).max(0)[None]
        for o in range(2):
            ref = -0.5 * (chi[:, o, s] * X).sum(1)
            bound = 2 * _dot_bound(aX, chi[:, o, s], 2 * n + 20) + (lost * np.abs(chi[:, o, s])).sum(1) + 1e-300
            assert np.all(np.abs(ehf[o, s] - ref) <= bound)
        B = -0.5 * sum(w[o, s][:, None] * chi[:, o, s] for o in range(2))
        aB = 0.5 * sum(np.abs(w[o, s][:, None] * chi[:, o, s]) for o in range(2))
        size = np.abs(ao).T @ aB
        bound = (N + 200) * U * size + N * 2.0 ** -55 * np.abs(ao).max(0)[:, None] * aB.max(0)[None] + 1e-300
        assert np.all(np.abs(fock[s] - ao.T @ B) <= bound)


def test_tiny_products(E):
    """Products down to the smallest normal numbers, in every column alike: off by the digits' 2^-57 and FP64 roundings
    as above, and by 2^-1022 for each product that FP64 would have kept as a denormal number."""
    n, N = 70, 200
    g = np.random.default_rng(5)
    ao = g.uniform(1, 2, (N, n)) * 10.0 ** g.uniform(-308, -280, N)[:, None]
    D, chi = g.standard_normal((2, n, n)), g.standard_normal((N, 1, 2, n))
    ehf = E.hf_energy_density(*(torch.as_tensor(v, device="cuda") for v in (ao, D, chi))).cpu().numpy()
    for s in range(2):
        aX = np.abs(ao) @ np.abs(D[s])
        bound = 2 * _dot_bound(aX, chi[:, 0, s], 2 * n + 20) + n * (2.0 ** -57 * np.abs(ao).max(1) * np.abs(
            D[s]).max() + 2.0 ** -1022) * np.abs(chi[:, 0, s]).sum(1)
        assert np.all(np.abs(ehf[0, s] + 0.5 * (chi[:, 0, s] * (ao @ D[s])).sum(1)) <= bound)


def test_gemms_past_one_slab(E):
    """The tall GEMMs hold the digits of about 512 MB at a time: 150,000 rows of a layer of width 256, 75,000 points of an
    exchange Fock term of 200 AOs.  Against float64 products on the GPU; rows and elements as above."""
    import graddft_gb300 as G
    import oracle as O
    from graddft_gb300 import synthetic

    rows, width = 160_001, 256
    p = synthetic.glorot_params(layer_widths=(width,), seed=3)
    x = torch.as_tensor(np.random.default_rng(4).standard_normal((rows, 11)), device="cuda")
    got = G.DM21(layer_widths=(width,)).apply(p, x)
    tp = {"params": {k: {kk: torch.as_tensor(v) for kk, v in d.items()} for k, d in p["params"].items()}}
    for part in (slice(0, 300), slice(149_000, 151_000), slice(rows - 300, rows)):  # the first slab's end among them
        assert torch.max(torch.abs(got[part].cpu() - O.dm21_network(tp, x[part].cpu(), n_layers=1))) <= 1e-13
    N, n = 80_001, 200
    g = torch.Generator(device="cuda").manual_seed(5)
    new = lambda *s: torch.randn(s, dtype=torch.float64, device="cuda", generator=g)  # noqa: E731
    ao, chi, w = new(N, n), new(N, 1, 2, n), new(1, 2, N)
    fock = E.hf_fock(ao, chi, w)
    for s in range(2):
        B = -0.5 * w[0, s][:, None] * chi[:, 0, s]
        # w's octaves move up to 2^3 from one operand to the other here: 2^-56 of the products of the scaled maxima.
        t = torch.exp2(torch.floor(torch.floor(torch.log2(w[0].abs().amax(0))) / 2))[:, None]
        lost = N * 2.0 ** -56 * (ao * t).abs().amax(0)[:, None] * (B / t).abs().amax(0)[None]
        bound = (N + 200) * U * (ao.abs().T @ B.abs()) + lost
        assert bool((torch.abs(fock[s] - ao.T @ B) <= bound).all())


@pytest.mark.parametrize("value", [2.0 ** 460, np.inf, np.nan])
def test_exchange_left_to_the_plain_kernels(E, value):
    """One AO value past the digits' range (2^450) or not finite: the plain kernels' sums and IEEE's pattern."""
    n, N = 70, 300
    g = np.random.default_rng(8)
    ao, D, chi, w = (g.standard_normal(s) for s in ((N, n), (2, n, n), (N, 1, 2, n), (1, 2, N)))
    ao[17, 5] = value
    c = lambda x: torch.as_tensor(x, device="cuda")  # noqa: E731
    ehf, fock = E.hf_energy_density(c(ao), c(D), c(chi)).cpu().numpy(), E.hf_fock(c(ao), c(chi), c(w)).cpu().numpy()
    for s in range(2):
        B = -0.5 * w[0, s][:, None] * chi[:, 0, s]
        with np.errstate(invalid="ignore"):
            refs = (ehf[0, s], -0.5 * (chi[:, 0, s] * (ao @ D[s])).sum(1), (np.abs(chi[:, 0, s]) * (np.abs(ao) @ np.abs(
                D[s]))).sum(1)), (fock[s], ao.T @ B, np.abs(ao).T @ np.abs(B))
        for got, ref, size in refs:
            ok = np.isfinite(size)
            assert np.all(np.abs(got[ok] - ref[ok]) <= 2 * (N + n) * U * size[ok])
            assert not np.isfinite(got[~ok]).any()


@pytest.mark.parametrize("what", ["ao", "rdm1", "pot"])
def test_past_the_digits_range(E, what):
    """A finite value past 2^450: density and V_xc come from the plain kernels, finite and right."""
    n, N = 40, 300
    ao, g1, g2, D, pot = _tables(n, N, 11)
    {"ao": ao, "rdm1": D[0], "pot": pot[0]}[what].flat[7] = 2.0 ** 460
    r = _resident(E, ao, g1, g2)
    rho = r.density(D)["rho"].cpu().numpy()
    v = r.vxc_from_potentials(pot).cpu().numpy()
    lap = g2.sum(-1)
    for s in range(2):
        size = ((np.abs(ao) @ np.abs(D[s])) * np.abs(ao)).sum(1)
        lost = n * 2.0 ** -56 * np.abs(ao).max(1) * np.abs(D[s]).max() * np.abs(ao).sum(1)  # where the digits serve
        assert np.all(np.abs(rho[:, s] - ((ao @ D[s]) * ao).sum(1)) <= 4 * n * U * size + lost + 1e-290)
        c = pot[s][..., None]
        Q = c[0] * ao + sum(c[1 + j] * g1[..., j] for j in range(3)) + c[4] * lap
        aQ = np.abs(c[0] * ao) + sum(np.abs(c[1 + j] * g1[..., j]) for j in range(3)) + np.abs(c[4] * lap)
        ref, size = ao.T @ Q, np.abs(ao).T @ aQ
        lost = np.abs(ao).max(0)[:, None] * aQ.max(0)[None]
        for j in range(3):
            K = c[5] * g1[..., j]
            ref += g1[..., j].T @ K
            size += np.abs(g1[..., j]).T @ np.abs(K)
            lost += np.abs(g1[..., j]).max(0)[:, None] * np.abs(K).max(0)[None]
        assert np.all(np.abs(v[s] - ref) <= (N + 400) * U * size + N * 2.0 ** -52 * np.maximum(lost, lost.T) + 1e-290)


@pytest.mark.parametrize("n,N", [(24, 400), (115, 300), (400, 120)])
def test_error_against_longer_sums(E, n, N):
    """The rounding error in itself, against sums in numpy's longer type (64 or 113 bits), as the root mean square over
    the points of the error relative to the sum of the terms' sizes.

    Independent roundings of up to half a unit (U / sqrt 3 in the mean square): one of each X, the n / 8 + 11 additions
    of a feature, and for V the additions of its partial sums, of which there are at most ten at these sizes."""
    g = np.random.default_rng(n)
    ao, g1, g2 = (g.standard_normal((N, n) + s) for s in ((), (3,), (3,)))
    q = np.linalg.qr(g.standard_normal((2, n, n)))[0][:, :, :max(1, n // 8)]
    D = q @ q.transpose(0, 2, 1)
    pot = g.standard_normal((2, 6, N))
    r = _resident(E, ao, g1, g2)
    out, v = r.density(D), r.vxc_from_potentials(pot).cpu().numpy()
    L = np.longdouble
    A, G, lap, limit = ao.astype(L), g1.astype(L), g2.sum(-1), U * (1 + np.sqrt((n / 8 + 12) / 3))
    rms = lambda got, ref, size: float(np.sqrt(np.mean(((got - ref) / size) ** 2)))  # noqa: E731
    for s in range(2):
        Dl = D[s].astype(L)
        X, aX = A @ Dl, np.abs(ao) @ np.abs(D[s])
        kin = sum(((G[..., j] @ Dl) * G[..., j]).sum(1) for j in range(3))
        akin = sum(((np.abs(g1[..., j]) @ np.abs(D[s])) * np.abs(g1[..., j])).sum(1) for j in range(3))
        o = {k: t[:, s].cpu().numpy() for k, t in out.items()}
        assert rms(o["rho"], (X * A).sum(1), (aX * np.abs(ao)).sum(1)) <= limit
        for j in range(3):
            assert rms(o["grad_rho"][:, j], 2 * (X * G[..., j]).sum(1), 2 * (aX * np.abs(g1[..., j])).sum(1)) <= limit
        assert rms(o["tau"], kin / 2, akin / 2) <= limit
        assert rms(o["lapl"], 2 * kin + 2 * (X * lap.astype(L)).sum(1), 2 * akin + 2 * (aX * np.abs(lap)).sum(1)) <= limit
        c = pot[s].astype(L)[..., None]
        each = [c[0] * A, *(c[1 + j] * G[..., j] for j in range(3)), c[4] * lap.astype(L)]
        ref, size = A.T @ sum(each), np.abs(ao).T @ sum(np.abs(t).astype(float) for t in each)
        for j in range(3):
            ref = ref + G[..., j].T @ (c[5] * G[..., j])
            size += np.abs(g1[..., j]).T @ np.abs(c[5] * G[..., j]).astype(float)
        assert rms(v[s], ref, size) <= U * (1 + np.sqrt((5 + 10) / 3))
