"""PathModel's gather kernel and its adjoint against the torch expressions they stand in for (PathModel.coords): every form
of box, revisited absorbers, negative indices, paths of mixed length, atoms that no path holds.  The coordinates are the
same operations (a general cell's two products may round differently: 1e-14 A); the gradient is the same sum in another
order (1e-13 of the largest)."""
import numpy as np
import pytest
import torch

from tests.fixtures import phase

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("box", [None, 9.0, (8.0, 9.0, 10.0), ((8.0, 0.3, 0.0), (0.0, 9.0, 0.5), (0.7, 0.0, 10.0))],
                         ids=["none", "cubic", "edges", "cell"])
@pytest.mark.parametrize("counts", [{2: 1}, {2: 5, 4: 40, 3: 9}, {9: 700}])
def test_gather_and_scatter(box, counts):
    from feffgpu_b200 import GPUPathStage
    from feffgpu_b200.model import PathModel, _Gather
    P = phase("cfg4_fe_phase")
    st = GPUPathStage(P, device="cuda")
    rng = np.random.default_rng(3)
    N = 20
    pos = rng.uniform(0, 9.0, (N, 3))
    groups = []
    for nleg, B in counts.items():
        at = np.zeros((B, nleg), int)
        at[:, 0] = rng.integers(0, 3, B)
        for j in range(1, nleg):
            at[:, j] = (at[:, j - 1] + rng.integers(1, 15, B)) % 16      # atoms 16.. unused
        if nleg > 3:
            at[:, 2] = at[:, 0]                                          # through the absorber
        at[0, -1] -= N                                                   # the same atom, counted from the end
        ip = np.ones((B, nleg), int)
        ip[:, 0] = 0
        groups.append((at, ip, None, None))
    m = PathModel(st, groups, pos, nrows=1, box=None if box is None else np.asarray(box) if np.ndim(box) else box)
    x = torch.tensor(pos + rng.normal(0, 0.1, pos.shape), device="cuda", requires_grad=True)
    got, ref = _Gather.apply(x, m), m.coords(x)
    assert (got - ref).abs().max() <= (1e-14 if np.ndim(box) else 0.0)
    w = torch.randn(got.shape, dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(1))
    g0, = torch.autograd.grad((got * w).sum(), x)
    g1, = torch.autograd.grad((ref * w).sum(), x)
    assert (g0 - g1).abs().max() <= 1e-13 * g1.abs().max()
    assert torch.all(g0[16:] == 0)


def test_a_model_without_paths_has_zero_rows_and_gradient():
    from feffgpu_b200 import GPUPathStage
    from feffgpu_b200.model import PathModel
    st = GPUPathStage(phase("cfg4_fe_phase"), device="cuda")
    m = PathModel(st, [(np.zeros((0, 3), int), np.zeros((0, 3), int))], np.eye(4, 3), nrows=2)
    x = torch.tensor(np.eye(4, 3), device="cuda", requires_grad=True)
    q = torch.arange(1, 12, dtype=torch.float64, device="cuda")
    rows = m.rows(x, q, st.linear_matrix(q.cpu().numpy()).double())
    assert rows.shape == (2, 11) and torch.all(rows == 0)
    g, = torch.autograd.grad(rows.sum(), x)
    assert g.shape == (4, 3) and torch.all(g == 0)


def test_out_of_range_atoms_are_refused():
    from feffgpu_b200 import GPUPathStage
    from feffgpu_b200.model import PathModel
    st = GPUPathStage(phase("cfg4_fe_phase"), device="cuda")
    for bad in (4, -5):
        with pytest.raises(IndexError):
            PathModel(st, [(np.array([[0, bad]]), np.array([[0, 1]]))], np.eye(4, 3), nrows=1)
