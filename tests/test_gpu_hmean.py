"""The plain form's horizontal mean of w: bit for bit the reference's chain of
rounded additions over the interior columns, whatever the sums do -- grow,
cancel, pass zero and powers of two, round half-way cases, overflow -- on
grids on both sides of every change of method (1280 and 8192 columns), ragged
segments among them.  The solve leaves w - mean in the outermost ghost plane
of w, which it corrects by nothing else.  Tolerance: none (equality)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GRIDS = [(3, 3, 3), (16, 16, 5), (40, 32, 7), (3, 427, 40), (32, 32, 26), (41, 25, 4), (64, 64, 3), (63, 65, 7), (90, 91, 3),
         (91, 91, 27), (96, 101, 6), (128, 130, 3)]
KINDS = ["turbulent", "random", "positive", "integers", "halves", "cancel", "scales", "zeros", "tiny", "nonfinite"]


def _columns(kind, n, rng):
    x = rng.standard_normal(n)
    if kind == "turbulent":
        return np.convolve(x, np.ones(9), mode="same")
    if kind == "positive":
        return np.abs(x)
    if kind == "integers":
        return np.rint(8 * x)
    if kind == "halves":  # ties: odd multiples of half the sum's unit, growing sums
        return np.rint(4 * x) * 2.0 ** -53 + rng.integers(0, 2, n) * 2.0 ** -52 + (np.arange(n) == 0)
    if kind == "cancel":
        return np.where(np.arange(n) % 2 == 0, x, -np.roll(x, 1))
    if kind == "scales":
        return x * 10.0 ** rng.integers(-12, 12, n)
    if kind == "zeros":
        return np.where(rng.random(n) < 0.9, -0.0, 0.0)
    if kind == "waves":  # sums that cancel every 64 columns: runs of segments added one by one
        return np.sin(2.0 * np.pi * np.arange(n) / 64.0)
    if kind == "returns":  # sums that come back to small values, exactly or nearly, from many binades
        x *= 2.0 ** rng.integers(-6, 6, n)
        run = 0.0
        for i in range(n):
            if rng.random() < 0.05:
                x[i] = -float(np.float32(run)) if rng.random() < 0.7 else -run
            run += x[i]
        return x
    if kind == "bursts":  # such runs between segments that move at once
        return np.where(np.arange(n) // 700 % 2 == 0, np.sin(2.0 * np.pi * np.arange(n) / 64.0), np.abs(x))
    if kind == "tiny":
        return x * 2.0 ** -1060
    if kind == "nonfinite":
        x[n // 2] = np.inf
    return x


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("grid", GRIDS, ids=lambda g: "x".join(map(str, g)))
def test_mean_equals_the_serial_chain(grid, kind):
    import torch
    from helpers import gpu_sim, host_case
    nl, rs, f = host_case(case="dry_cbl", nx=4, ny=4, nz=grid[2], dx=50.0, dy=50.0, dz=50.0)
    nl["grid"].update(nx=grid[0], ny=grid[1])
    sim = gpu_sim(nl, rs, {})
    Gr, PV = sim.Gr, sim.PV
    rng = np.random.default_rng(3)
    g = Gr.dims.gw
    w = rng.standard_normal(Gr.shape)
    for k in range(w.shape[2]):
        w[g:-g, g:-g, k] = _columns(kind, grid[0] * grid[1], rng).reshape(grid[0], grid[1])
    w[-1] = 0.0
    with np.errstate(all="ignore"):
        want = np.add.accumulate(w[g:-g, g:-g].reshape(-1, w.shape[2]), axis=0)[-1] + 0.0
        want = 0.0 - want * (1.0 / (grid[0] * grid[1]))
    PV.get_variable_array("w", Gr).copy_(torch.as_tensor(w))
    sim.Pr.solve(Gr, sim.RS, sim.DV, PV)
    got = PV.get_variable_array("w", Gr)[-1].cpu().numpy()
    np.testing.assert_array_equal(got, np.broadcast_to(want, got.shape))


@pytest.mark.parametrize("kind", ["waves", "bursts", "returns"])
@pytest.mark.parametrize("grid", [(41, 64, 5), (64, 64, 3), (90, 91, 3), (96, 101, 6), (128, 130, 3), (150, 64, 28)],
                         ids=lambda g: "x".join(map(str, g)))
def test_mean_of_cancelling_columns(grid, kind):
    test_mean_equals_the_serial_chain(grid, kind)
