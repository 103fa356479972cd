"""Inverse iteration on tridiagonals whose eigenvalues come in clusters of
every length: one, a few, all of them; around the warp, at the largest size
that runs from shared memory (512) and just past it.

Bounds as for the other tridiagonals (tests/test_gpu_lanczos.py): a vector
of inverse iteration from a random start has a residual of a few k units of
2^-53 of |T| (5e-14 at k = 513; 1e-12 allows for the start vector's component
growing less than its norm), and a Gram-Schmidt pass after each of three
solves leaves overlaps of 2^-53 times the cluster's length over the gap the
shifts open, below 1e-9."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("needs a CUDA device", allow_module_level=True)

from parsec_python_b200 import gpu  # noqa: E402

DEV = torch.device("cuda", 0)


def _matrix(kind, k):
    if kind == "single":
        return np.arange(k, dtype=float), np.full(k, 0.3)
    if kind == "pairs":
        return np.repeat(np.arange((k + 1) // 2, dtype=float), 2)[:k], np.full(k, 1e-9)
    if kind == "blocks":
        return np.repeat([1.0, 2.0, 3.5], (k + 2) // 3)[:k], np.full(k, 1e-12)
    return np.zeros(k), np.zeros(k)


@pytest.mark.parametrize("k", [1, 2, 31, 33, 64, 512, 513])
@pytest.mark.parametrize("kind", ["single", "pairs", "blocks", "zero"])
def test_clusters(kind, k):
    if kind in ("blocks", "zero") and k > 64:
        k = {512: 70, 513: 96}[k]           # (long clusters: the passes grow with the square)
    d, e = _matrix(kind, k)
    T = np.diag(d) + np.diag(e[:k - 1], 1) + np.diag(e[:k - 1], -1)
    ab = np.zeros(2 * k)
    ab[0::2], ab[1::2] = d, e
    ctx = gpu.GridContext({"nx": 4, "ny": 4, "nz": 4, "h": 1.0, "radius": 1.0}, 8)
    abd = torch.from_numpy(ab).to(DEV)
    ev = torch.empty(k, dtype=torch.float64, device=DEV)
    Z = torch.empty(k, k, dtype=torch.float64, device=DEV)
    ctx.call("psc_tridiag_eig", gpu._p(abd), k, k, gpu._p(ev), gpu._p(Z), k, gpu._stream())
    w, z = ev.cpu().numpy(), Z.cpu().numpy().T
    tn = max(np.abs(T).sum(1).max(), 1e-100)
    assert np.abs(w - np.linalg.eigvalsh(T)).max() <= 8e-15 * k * tn
    assert np.abs(T @ z - z * w).max() <= 1e-12 * tn
    assert np.abs(z.T @ z - np.eye(k)).max() < 1e-9
