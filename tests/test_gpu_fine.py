"""The fine-grid kernels of the drop-in calls (a block per path) where their block's loops and shared memory change shape:
one point, counts around the 128 threads, and the last one whose backward fits 48 KB of shared memory and the next.

Against the same sums by torch in FP64, inputs equal: in FP64 only the order of the sums differs (1e-10 of the largest
component), in the mixed form the sines are FP32 of an FP64 argument and the results are rounded to FP32 (1e-5)."""
import math

import pytest
import torch

from tests.fixtures import phase

pytestmark = pytest.mark.gpu
P = phase("case_L001")
E = int(P.ne1)


@pytest.mark.parametrize("dtype", [torch.complex64, torch.complex128])
@pytest.mark.parametrize("NK", [1, 127, 129, 3072 - E, 3073 - E])
def test_chi_fine_and_its_gradient(dtype, NK):
    from feffgpu_b200 import GPUPathStage
    st = GPUPathStage(P, device="cuda", dtype=dtype)
    B = 7
    gen = torch.Generator().manual_seed(NK)
    ph = torch.cumsum(0.4 + 0.5 * torch.rand(B, E, generator=gen, dtype=torch.float64), 1)
    c = torch.polar(0.5 + torch.rand(B, E, generator=gen, dtype=torch.float64), ph).to(dtype)
    rf = (2.0 + 3.0 * torch.rand(B, generator=gen, dtype=torch.float64)).to(st.rdtype)
    q = torch.linspace(0.5, 15.0, NK, dtype=torch.float64).to(st.rdtype)
    S = st.linear_matrix(q.double().numpy()).to(st.rdtype).cpu()
    g = torch.randn(B, NK, generator=gen, dtype=torch.float64).to(st.rdtype)

    def run(c, rf, chi):
        c, rf = c.clone().requires_grad_(True), rf.clone().requires_grad_(True)
        out = chi(c, rf)
        gc, gr = torch.autograd.grad(out, (c, rf), g.to(out.device, out.dtype))
        return [v.detach().cpu() for v in (out.double(), torch.view_as_real(gc).double(), gr.double())]

    def oracle(c, rf):
        ang = torch.angle(c)
        d = ang[:, 1:] - ang[:, :-1]
        turns = torch.cumsum(-torch.round(d.detach() / (2 * math.pi)), 1) * 2 * math.pi
        pha = torch.cat([ang[:, :1], ang[:, 1:] + turns], 1)
        return (c.abs() @ S.double().T) * torch.sin(pha @ S.double().T + 2 * q.double() * rf[:, None])

    got = run(c.cuda(), rf.cuda(), lambda a, b: st.chi_fine(a, b, q.cuda(), S.cuda()))
    ref = run(c.to(torch.complex128), rf.double(), oracle)
    tol = 1e-10 if dtype == torch.complex128 else 1e-5
    for a, b in zip(got, ref):
        assert torch.allclose(a, b, rtol=0, atol=tol * float(b.abs().max()))


@pytest.mark.parametrize("dtype", [torch.complex64, torch.complex128])
@pytest.mark.parametrize("NK", [1, 33, 401])
def test_a_path_has_the_same_bits_whatever_the_number_of_paths(dtype, NK):
    """Calls of 96 paths per SM and more take a warp per path instead of a block: the same operations in the same order."""
    from feffgpu_b200 import GPUPathStage
    st = GPUPathStage(P, device="cuda", dtype=dtype)
    B = 96 * torch.cuda.get_device_properties(0).multi_processor_count + 3
    gen = torch.Generator("cuda").manual_seed(NK)
    c = torch.view_as_complex(torch.randn(B, E, 2, device="cuda", dtype=st.rdtype, generator=gen))
    rf = 2.0 + 3.0 * torch.rand(B, device="cuda", dtype=st.rdtype, generator=gen)
    q = torch.linspace(0.5, 15.0, NK, dtype=torch.float64)
    S = st.linear_matrix(q.numpy())
    got = st.chi_fine(c, rf, q, S)
    parts = [st.chi_fine(c[i:i + 5000], rf[i:i + 5000], q, S) for i in range(0, B, 5000)]
    assert torch.isfinite(got).all() and torch.equal(got, torch.cat(parts))
