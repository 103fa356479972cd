"""Reductions that end in the launch's last CTA (LDA sums, potential update,
dot products) and the block-wide Fermi bisection, at the sizes where their
splits change: one CTA, whole and partial CTAs, more points than threads."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - collected on CPU runs
    pytest.skip("needs a CUDA device", allow_module_level=True)

from parsec_python_b200 import gpu  # noqa: E402

DEV = torch.device("cuda", 0)
EPS = np.finfo(float).eps
# 1 point; one short CTA; one full CTA of points; several; more than 592 x 256 points
GRIDS = [(1, 1, 1), (5, 5, 5), (16, 16, 1), (17, 16, 1), (41, 25, 1), (61, 55, 47)]


def _ctx(dims):
    return gpu.GridContext({"nx": dims[0], "ny": dims[1], "nz": dims[2], "h": 0.4, "radius": 1.0}, 2)


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).to(DEV)


@pytest.mark.parametrize("dims", GRIDS)
def test_xc_and_update_sums(dims):
    ctx = _ctx(dims)
    n = ctx.n
    rng = np.random.default_rng(n)
    rho = np.exp(rng.uniform(-12, 3, n))
    rho[rng.integers(0, n)] *= 2.0
    for _ in range(2):   # twice: the arrival counter is back at zero after a launch
        vxc, out = gpu.lda_xc(ctx, _dev(rho))
    ref_v, ref_e = O.exc_nspn(0.4, rho)
    o = out.cpu().numpy()
    assert np.abs(vxc.cpu().numpy() - ref_v).max() <= 1e-13 * np.abs(ref_v).max()
    # a sum of n terms of one sign: any order is within n eps of the exact one
    assert abs(o[0] - ref_e) <= 2 * n * EPS * abs(ref_e) + 1e-13 * abs(ref_e)
    assert o[1] == rho.max() and o[2] == rho.min()
    f = [rng.standard_normal(n) for _ in range(5)]
    pot_new, d, sums = gpu.scf_update(ctx, *(_dev(v) for v in f[:4]), _dev(rho), _dev(f[4]))
    pn = f[0] + 0.5 * f[1] + f[2] + f[3]
    terms = [(pn - f[4]) ** 2, pn ** 2, rho * (f[2] + f[3]), rho * f[1]]
    assert np.abs(pot_new.cpu().numpy() - pn).max() <= 4 * EPS * np.abs(pn).max()
    assert np.abs(d.cpu().numpy() - (pn - f[4])).max() <= 8 * EPS * max(np.abs(pn).max(), np.abs(f[4]).max())
    for got, t in zip(sums.cpu().numpy(), terms):
        assert abs(got - t.sum()) <= 2 * (n + 8) * EPS * np.abs(t).sum()
    out1 = ctx.empty(1)
    a, b = _dev(f[0]), _dev(f[1])
    ctx.call("psc_dot", gpu._p(a), gpu._p(b), n, gpu._p(out1), gpu._stream())
    assert abs(float(out1) - f[0] @ f[1]) <= 2 * n * EPS * np.abs(f[0] * f[1]).sum()


def test_xc_extremes_propagate_nan_from_any_cta():
    ctx = _ctx((61, 55, 47))
    for at in (0, 77_777, ctx.n - 1):
        rho = np.full(ctx.n, 0.3)
        rho[at] = np.nan
        _, out = gpu.lda_xc(ctx, _dev(rho))
        assert np.isnan(out.cpu().numpy()[1:]).all()


@pytest.mark.parametrize("n", [1, 31, 32, 33, 292, 1024, 1500])
def test_occupations_by_state_count(n):
    ctx = _ctx((5, 5, 5))
    lam = np.sort(np.random.default_rng(n).uniform(-1.0, 0.5, n))
    ne = 2.0 * max(1, int(0.7 * n)) if n > 1 else 1.5
    ef, occ = gpu.occupations(ctx, _dev(lam), 500.0, ne, 1e-6)
    ref_ef, ref_occ = O.occupations(lam, 500.0, ne, 1e-6)
    # the bisections take the same steps: equal up to the rounding of exp
    assert abs(float(ef) - ref_ef) <= 1e-12
    assert np.abs(occ.cpu().numpy() - ref_occ).max() <= 1e-9


@pytest.mark.parametrize("dims", [(5, 5, 5), (17, 16, 3), (61, 55, 47)])
def test_mixer_history_groups_and_restart(dims):
    """Thirteen secant columns (three groups of four and one over), a restart,
    and four more, against the oracle's msecant1."""
    ctx = _ctx(dims)
    rng = np.random.default_rng(sum(dims))
    ours, ref = gpu.Mixer(ctx, 40), O.MSecant1()
    for i in range(19):
        f = rng.standard_normal(ctx.n) * 0.7 ** i
        if i >= 14:
            f *= 1e3      # |f| of the call before < 0.1 |f|: restart at i = 14
        x = 1.0 + 0.5 ** i * rng.standard_normal(ctx.n)
        got, m = ours(_dev(x), _dev(f))
        want, m_ref = ref(x, f)
        assert m == m_ref and (i != 14 or m == 0)
        # independent columns: the secant equations are well conditioned
        assert np.abs(got.cpu().numpy() - want).max() <= 1e-10 * np.abs(want).max()
