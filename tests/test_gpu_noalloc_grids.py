"""dasha_current_noalloc on grids of every alignment and the smallest it takes, against the equations in
FP64 numpy: curl of the perturbation by the exact five-point weights, wall rows, four passes with the
radial coefficient.  The last grid's spacings differ by more than the device-made tables take, so that
its tables come from the host.  Tolerance: a curl of O(1/h) sums of O(1) values and 4 smoothing passes, all
FP64, agree to a few hundred ulp of the result's scale: 1e-12."""
import numpy as np
import pytest

from dasha_b200 import capi, harris

pytestmark = pytest.mark.gpu


def _current(db, x, y, z):
    ax = {0: 2, 1: 1, 2: 0}
    C = {0: harris.deriv_coefficients(x, True), 1: harris.deriv_coefficients(y, True), 2: harris.deriv_coefficients(z, False)}

    def shape(v, d):
        return v.reshape([-1 if ax[d] == q else 1 for q in range(3)])

    def D(f, d):
        r = lambda s: np.roll(f, -s, ax[d])  # noqa: E731
        a, b, c, e = (shape(v, d) for v in C[d])
        return a * (r(1) - f) + b * (f - r(-1)) + c * (r(2) - f) + e * (f - r(-2))

    def rows(f):
        g = np.zeros_like(f)
        g[2:-2] = f[2:-2]
        g[1], g[-2] = 0.5 * f[2], 0.5 * f[-3]
        return g

    w = {}
    for d, c in enumerate((x, y, z)):
        L = c[-1] - c[0] + c[1] - c[0]
        e = np.concatenate([[c[-1] - L], c, [c[0] + L]])
        w[d] = [shape(2 * (e[2:] - e[1:-1]) / (e[2:] - e[:-2]), d), shape(2 * (e[1:-1] - e[:-2]) / (e[2:] - e[:-2]), d)]
    r = np.sqrt(shape(x, 0) ** 2 + shape(y, 1) ** 2 + shape(z, 2) ** 2)
    cr = 1 / 32 + 3 / 64 * (1 + np.tanh((r - 3) / 3))
    J = [rows(f) for f in (D(db[2], 1) - D(db[1], 2), D(db[0], 2) - D(db[2], 0), D(db[1], 0) - D(db[0], 1))]
    for _ in range(4):
        J = [rows(f + cr * sum((np.roll(f, -1, ax[d]) - f) * w[d][0] - (f - np.roll(f, 1, ax[d])) * w[d][1] for d in range(3)))
             for f in J]
    return np.stack(J)


@pytest.mark.parametrize("grid", [(5, 5, 7), (7, 9, 8), (33, 6, 13), (128, 64, 100), (16, 8, 12, 1e4)],
                         ids=lambda g: "x".join(map(str, g)))
def test_noalloc_current_on_any_grid(grid):
    import torch
    x, y, z = harris.make_grid(*grid[:3], True)
    if len(grid) == 4:
        z = np.concatenate([z[:6], z[5] + grid[3] * (z[6:] - z[5])])   # one spacing 1e4 times its neighbour
    db = np.random.default_rng(2).standard_normal((3, z.size, y.size, x.size))
    dev = torch.tensor(db, device="cuda")
    out = torch.full_like(dev, float("nan"))
    assert capi.current_noalloc(x, y, z, dev.data_ptr(), out.data_ptr(), 0) == capi.OK
    torch.cuda.synchronize()
    ref = _current(db, x, y, z)
    assert np.abs(out.cpu().numpy() - ref).max() <= 1e-12 * np.abs(ref).max()
