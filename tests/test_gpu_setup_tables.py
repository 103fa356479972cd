"""The table form of the SAD setup and the projector tables built on the
device, where their look-ups and prefix sums have edges: distances of zero,
beyond the last bucket and in the clamped tail, species changing from atom to
atom, grids of fewer points than a scan block and of more blocks than one
scan pass takes."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - collected on CPU runs
    pytest.skip("needs a CUDA device", allow_module_level=True)

from parsec_python_b200 import gpu  # noqa: E402
from parsec_python_b200.inputs import ElementTable, pseudo_tables  # noqa: E402

DEV = torch.device("cuda", 0)


def _domain(nx, ny, nz, h):
    return {"nx": nx, "ny": ny, "nz": nz, "h": h, "radius": 0.5 * h * (nx - 1)}


@pytest.mark.parametrize("dims,h", [((3, 2, 1), 0.4), ((9, 8, 7), 0.3), ((16, 17, 5), 0.9), ((11, 11, 11), 25.0)])
def test_sad_setup_is_bit_exact(dims, h):
    dom = _domain(*dims, h)
    rng = np.random.default_rng(int(100 * h))
    r = dom["radius"]
    # one atom on a grid point (r = 0 there), the others anywhere, some outside
    atoms = [{"typ": t, "coord": np.vstack([[-r, -r, -r] if i == 0 else rng.uniform(-r, 1.3 * r, 3), rng.uniform(-r, r, (2, 3))])}
             for i, t in enumerate(("Si", "H", "C", "O"))]
    ctx = gpu.GridContext(dom, 8)
    rho0, hpot0, ppot, info = gpu.sad_setup(ctx, atoms, ElementTable(), pseudo_tables())
    want = O.pseudo_diag(dom, atoms, O.load_elements(), O.load_tables())
    for got, ref in zip((rho0, hpot0, ppot), want[:3]):
        assert np.array_equal(got.cpu().numpy(), ref)
    assert info["electron_count_initial"] == want[3]["electron_count_initial"]


@pytest.mark.parametrize("dims,h", [((7, 6, 5), 0.9), ((33, 31, 29), 0.35), ((90, 84, 82), 0.3)])
def test_projector_tables_and_their_covers(dims, h):
    dom = _domain(*dims, h)
    rng = np.random.default_rng(dims[0])
    mid = 0.5 * h * (np.array(dims) - dims[0])
    # close atoms whose balls overlap, one at a corner, one whose box is outside
    atoms = [{"typ": "Si", "coord": np.vstack([mid + rng.uniform(-1, 1, (4, 3)), [[-dom["radius"]] * 3]])},
             {"typ": "O", "coord": np.vstack([mid + rng.uniform(-1, 1, (2, 3)), mid + 50 * h * max(dims)])}]
    ctx = gpu.GridContext(dom, 8)
    proj = gpu.projector_setup(ctx, atoms, ElementTable(), pseudo_tables())
    projs = O.projectors(dom, atoms, O.load_elements(), O.load_tables())
    x = rng.standard_normal((ctx.n, 3))
    X = torch.from_numpy(np.ascontiguousarray(x.T)).to(DEV)
    got = []
    for _ in range(2):
        Y = torch.empty_like(X)
        ctx.call("psc_apply_nonlocal", 0, gpu._p(X), ctx.n, gpu._p(Y), ctx.n, 3, gpu._stream())
        got.append(Y.cpu().numpy())
        proj = gpu.projector_setup(ctx, atoms, ElementTable(), pseudo_tables())   # the tables again
    assert np.array_equal(got[0], got[1])       # the same order of entries every time
    ref = O.nonlocal_apply(projs, x)
    assert np.abs(got[0].T - ref).max() <= 1e-13 * np.abs(ref).max()
    off, idx, _, _ = proj.tables()
    assert proj.n_touched == len(np.unique(idx))
    assert all((np.diff(idx[a:b]) > 0).all() for a, b in zip(off[:-1], off[1:]))
