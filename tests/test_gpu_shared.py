"""The shared-matrix and staged forms of the fused stage and of the drop-in signal (csrc/fg_shared.cuh) against the
one-kernel form, which a call given only the head and the row sums as workspace (fg_chi_reduce) or none (fg_cchi) takes:
the same operations in the same order per value, so signals and rows are the same bits, over leg counts 2..9, revisits,
sizes around the rules, two sub-batches, and lists without any equal scatterers.  (The adjoints sum in another order.)"""
import ctypes as C

import numpy as np
import pytest
import torch

from tests.fixtures import phase

pytestmark = pytest.mark.gpu
DTYPES = [torch.complex64, torch.complex128]


def _list(nph, counts, atoms, seed=0):
    """Paths over few atoms (their scatterers repeat) as PathBatch groups; consecutive atoms differ, revisits allowed."""
    rng = np.random.default_rng(seed)
    pts = np.zeros((1, 3))
    while len(pts) <= atoms:                         # no two atoms closer than 1.8 A, as in matter
        x = rng.uniform(-4.0, 4.0, 3)
        if np.linalg.norm(pts - x, axis=1).min() > 1.8:
            pts = np.concatenate([pts, x[None]])
    pot = np.concatenate([[0], rng.integers(1, nph + 1, atoms)])
    groups = []
    for nleg, B in counts.items():
        seq = np.zeros((B, nleg), int)
        for j in range(1, nleg):
            last = j == nleg - 1
            lo = 1 if j == 1 or last else 0
            pick = rng.integers(lo, atoms + 1, B)
            while (bad := (pick == seq[:, j - 1])).any():
                pick[bad] = rng.integers(lo, atoms + 1, int(bad.sum()))
            seq[:, j] = pick
        groups.append((pts[seq], pot[seq], rng.uniform(1, 3, B), rng.integers(0, 3, B)))
    return groups


def _rows(st, b, q, S, shared, words=False):
    from feffgpu_b200 import _lib
    span = st._span(S)
    ps = st._paths_struct(b, b.coords, None)
    NK = int(q.shape[0])
    full = int(st._lib.fg_chi_reduce_workspace(st._h, C.byref(ps), NK))
    least = 256 + (16 * b.nrows * NK + 255) // 256 * 256
    ws = torch.empty(full if shared else least, dtype=torch.uint8, device="cuda")
    rows = torch.empty(b.nrows, NK, dtype=torch.float64, device="cuda")
    cc = torch.empty(b.n, st.E, dtype=st.cdtype, device="cuda")
    rf = torch.empty(b.n, dtype=torch.float64, device="cuda")
    _lib.check(st._lib.fg_chi_reduce(st._h, st.prec, C.byref(ps), NK, q.data_ptr(), S.data_ptr(), span.data_ptr(),
                                     rows.data_ptr(), cc.data_ptr(), rf.data_ptr(), ws.data_ptr(), ws.numel(),
                                     torch.cuda.current_stream().cuda_stream))
    return rows, cc, rf, full > least


def _same(a, b, tol):
    assert torch.isfinite(torch.view_as_real(b) if b.is_complex() else b).all()
    assert (a - b).abs().max() <= tol * b.abs().max()


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("case", ["cfg2_phase", "case_A014", "case_A009"])
@pytest.mark.parametrize("nk", [0, 161])
@pytest.mark.parametrize("counts", [{4: 1}, {2: 7, 3: 33, 4: 5}, {9: 40, 8: 3, 2: 1}, {6: 3000, 5: 2000, 3: 11}],
                         ids=["one", "few", "long", "many"])
def test_shared_form_equals_one_kernel_form(dtype, case, nk, counts):
    from feffgpu_b200 import GPUPathStage, PathBatch
    from feffgpu_b200.pad import resample_phase
    P = resample_phase(phase(case), np.linspace(0.0, 20.0, nk)) if nk else phase(case)
    st = GPUPathStage(P, device="cuda", dtype=dtype)
    b = PathBatch(_list(P.nph, counts, 7), nrows=3, device="cuda")
    q = torch.arange(1, 402, dtype=torch.float64, device="cuda") * 0.05
    S = st.linear_matrix(q.cpu().numpy()).double().contiguous()
    got, cc, rf, offered = _rows(st, b, q, S, True)
    ref, cr, rr, _ = _rows(st, b, q, S, False)
    # share_plan's rule at 2, 3 and 6 chunks of energies: classes, or the staged form from 4,096 (path, chunk) items
    assert offered == (nk > 0 or b.n > 4000 or st.ilinit > 1)
    assert torch.equal(cc, cr) and torch.isfinite(torch.view_as_real(cc)).all()
    assert torch.equal(got, ref)
    assert torch.equal(rf, rr)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("case", ["cfg2_phase", "case_A014", "case_A009"])
@pytest.mark.parametrize("counts", [{3: 2050}, {2: 4100}, {4: 2300, 3: 7, 2: 3}, {3: 32000, 2: 1001}],
                         ids=["short", "two", "four", "sub-batches"])
def test_staged_form_equals_one_kernel_form(dtype, case, counts):
    """The staged form (many paths on few energies): one sub-batch of 2^15 paths and two, rows that change from path to
    path, interpolation matrices of two entries a row and of many, more fine-grid points than the shared sums hold."""
    from feffgpu_b200 import GPUPathStage, PathBatch
    P = phase(case)
    st = GPUPathStage(P, device="cuda", dtype=dtype)
    b = PathBatch(_list(P.nph, counts, 7, seed=8), nrows=3, device="cuda")
    q = torch.arange(1, 402, dtype=torch.float64, device="cuda") * 0.05
    S = st.linear_matrix(q.cpu().numpy()).double().contiguous()
    got, cc, rf, offered = _rows(st, b, q, S, True)
    ref, cr, rr, _ = _rows(st, b, q, S, False)
    assert offered
    assert torch.equal(cc, cr) and torch.isfinite(torch.view_as_real(cc)).all()
    assert torch.equal(got, ref)
    assert torch.equal(rf, rr)
    if b.n < 3000:
        for nk in (35, 1300):
            qk = torch.linspace(0.5, 15.0, nk, dtype=torch.float64, device="cuda")
            D = torch.softmax(-(qk[:, None] - torch.linspace(0.5, 15.0, st.E, dtype=torch.float64, device="cuda")) ** 2, 1)
            D = torch.where(D > 1e-3, D, 0.0).contiguous()
            assert torch.equal(_rows(st, b, qk, D, True)[0], _rows(st, b, qk, D, False)[0])


@pytest.mark.parametrize("dtype", DTYPES)
def test_shared_form_over_two_sub_batches_and_without_sharing(dtype):
    """More paths than one sub-batch holds (2^18); and paths with no two scatterers alike, with which the call goes on in
    the staged form after it has counted them."""
    from feffgpu_b200 import GPUPathStage, PathBatch
    P = phase("case_A014")
    st = GPUPathStage(P, device="cuda", dtype=dtype)
    q = torch.arange(1, 21, dtype=torch.float64, device="cuda")
    S = st.linear_matrix(q.cpu().numpy()).double().contiguous()
    groups = _list(P.nph, {4: (1 << 18) - 3, 3: 9, 2: 4}, 6, seed=1)
    b = PathBatch(groups, nrows=3, device="cuda")
    got, cc, _, offered = _rows(st, b, q, S, True)
    ref, cr, _, _ = _rows(st, b, q, S, False)
    assert offered
    assert torch.equal(cc, cr) and torch.isfinite(torch.view_as_real(cc)).all()
    assert torch.equal(got, ref)
    rng = np.random.default_rng(2)
    own = [(c + np.where(np.arange(c.shape[1])[None, :, None] > 0, rng.normal(0, 0.05, c.shape), 0.0), i, d, r)
           for c, i, d, r in ((c[:9000], i[:9000], d[:9000], r[:9000]) for c, i, d, r in groups)]
    b = PathBatch(own, nrows=3, device="cuda")
    got, cc, _, _ = _rows(st, b, q, S, True)
    ref, cr, _, _ = _rows(st, b, q, S, False)
    assert torch.equal(cc, cr) and torch.isfinite(torch.view_as_real(cc)).all()
    assert torch.equal(got, ref)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("nleg,B", [(2, 5), (3, 1), (4, 700), (7, 9000), (9, 31)])
def test_drop_in_signal_with_and_without_scratch(dtype, nleg, B):
    from feffgpu_b200 import GPUPathStage, _lib
    P = phase("case_A014")
    st = GPUPathStage(P, device="cuda", dtype=dtype)
    c, ip, _, _ = _list(P.nph, {nleg: B}, 6, seed=3)[0]
    c = torch.tensor(c, device="cuda", dtype=st.rdtype)
    ip = torch.tensor(ip, device="cuda")
    got, rf = st.cchi(c, ip)
    ref = torch.empty_like(got)
    rr = torch.empty_like(rf)
    _lib.check(st._lib.fg_cchi(st._h, st.prec, B, nleg, c.data_ptr(), int(dtype == torch.complex128), ip.data_ptr(),
                               ref.data_ptr(), rr.data_ptr(), None, torch.cuda.current_stream().cuda_stream))
    assert torch.equal(got, ref) and torch.isfinite(torch.view_as_real(got)).all()
    assert torch.equal(rf, rr)


def _grads(st, b, q, S, shared, g, s2):
    """Fused backward's (grad_coords, grad_sigma2) from the one-kernel form's saved signals."""
    from feffgpu_b200 import _lib
    span, tspan = st._span(S), st._span(S, True)
    NK = int(q.shape[0])
    ps = st._paths_struct(b, b.coords, s2)
    _, cc, rf, _ = _rows(st, b, q, S, False)
    full = int(st._lib.fg_chi_reduce_backward_workspace(st._h, C.byref(ps), NK))
    up = lambda v: (v + 255) // 256 * 256  # noqa: E731
    least = 256 + up(b.n * st.E * 16) + up(b.n * 8) + up(b.n * 256)
    ws = torch.empty(full if shared else least, dtype=torch.uint8, device="cuda")
    gc = torch.empty_like(b.coords)
    gs = torch.empty(b.n, dtype=torch.float64, device="cuda")
    _lib.check(st._lib.fg_chi_reduce_backward(st._h, st.prec, C.byref(ps), NK, q.data_ptr(), S.data_ptr(),
                                              span.data_ptr(), tspan.data_ptr(), g.data_ptr(), cc.data_ptr(),
                                              rf.data_ptr(), gc.data_ptr(), gs.data_ptr(), ws.data_ptr(), ws.numel(),
                                              torch.cuda.current_stream().cuda_stream))
    return gc, gs, full > least


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("case,iorder", [("cfg2_phase", 2), ("case_A014", 2), ("case_A009", 2), ("cfg2_phase", 1),
                                         ("case_A014", 0)])
@pytest.mark.parametrize("counts", [{3: 1}, {2: 7, 3: 33, 4: 5}, {9: 40, 8: 3, 2: 1}, {6: 1500, 5: 500, 2: 9}],
                         ids=["one", "few", "long", "many"])
def test_shared_adjoint_equals_one_kernel_adjoint(dtype, case, iorder, counts):
    """The gradients of both forms: the shared one sums a class's derivative over the partial waves before a path's
    weights meet it, the other the weighted terms, so they agree to the rounding of such sums (of order 100 terms: 1e-5
    of the largest component in the mixed form, 1e-11 in FP64)."""
    from feffgpu_b200 import GPUPathStage, PathBatch
    from feffgpu_b200.pad import resample_phase
    P = resample_phase(phase(case), np.linspace(0.0, 20.0, 131))
    st = GPUPathStage(P, device="cuda", dtype=dtype, iorder=iorder)
    b = PathBatch(_list(P.nph, counts, 7, seed=4), nrows=3, device="cuda")
    q = torch.arange(1, 202, dtype=torch.float64, device="cuda") * 0.1
    S = st.linear_matrix(q.cpu().numpy()).double().contiguous()
    gen = torch.Generator("cuda").manual_seed(5)
    g = torch.randn(3, 201, dtype=torch.float64, device="cuda", generator=gen)
    s2 = 0.001 + 0.004 * torch.rand(b.n, dtype=torch.float64, device="cuda", generator=gen)
    got, gs, offered = _grads(st, b, q, S, True, g, s2)
    ref, rs, _ = _grads(st, b, q, S, False, g, s2)
    assert offered
    _same(got, ref, {torch.complex64: 1e-5, torch.complex128: 1e-11}[dtype])
    assert torch.equal(gs, rs)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("nleg,B", [(2, 5), (3, 1), (4, 700), (7, 5000)])
def test_drop_in_adjoint_with_and_without_scratch(dtype, nleg, B):
    from feffgpu_b200 import GPUPathStage, _lib
    P = phase("case_A014")
    st = GPUPathStage(P, device="cuda", dtype=dtype)
    c, ip, _, _ = _list(P.nph, {nleg: B}, 6, seed=6)[0]
    c = torch.tensor(c, device="cuda", dtype=st.rdtype)
    ip = torch.tensor(ip, device="cuda")
    gen = torch.Generator("cuda").manual_seed(7)
    g = torch.randn(B, st.E, 2, dtype=st.rdtype, device="cuda", generator=gen)
    gr = torch.randn(B, dtype=st.rdtype, device="cuda", generator=gen)
    got = st._cchi_backward(c, ip, torch.view_as_complex(g), gr)
    ref = torch.empty_like(got)
    ws = torch.empty(256, dtype=torch.uint8, device="cuda")
    _lib.check(st._lib.fg_cchi_backward(st._h, st.prec, B, nleg, c.data_ptr(), int(dtype == torch.complex128),
                                        ip.data_ptr(), g.data_ptr(), gr.data_ptr(), ref.data_ptr(), ws.data_ptr(), 256,
                                        torch.cuda.current_stream().cuda_stream))
    _same(got, ref, {torch.complex64: 1e-5, torch.complex128: 1e-11}[dtype])


@pytest.mark.parametrize("counts", [{6: 3000, 5: 1000, 2: 9}, {3: 33000}], ids=["classes", "staged"])
def test_forms_replay_in_a_graph(counts):
    """The shared and staged forms under stream capture: a replay with moved atoms finds its classes anew and gives the
    eager call's rows and gradients (the forward bit for bit; the adjoint's sums are in a fixed order too)."""
    from feffgpu_b200 import GPUPathStage, PathBatch
    from feffgpu_b200.pad import resample_phase
    P = resample_phase(phase("cfg2_phase"), np.linspace(0.0, 20.0, 131)) if 3 not in counts else phase("cfg2_phase")
    st = GPUPathStage(P, device="cuda")
    groups = _list(P.nph, counts, 7, seed=9)
    b = PathBatch(groups, nrows=3, device="cuda")
    q = torch.arange(1, 102, dtype=torch.float64, device="cuda") * 0.15
    S = st.linear_matrix(q.cpu().numpy()).double().contiguous()
    g = torch.randn(3, 101, dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(2))
    x = b.coords.clone().requires_grad_(True)

    def step():
        rows = st.chi_reduce(b, q, S, coords=x)
        return rows.detach(), torch.autograd.grad(rows, x, g)[0]

    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        step()
    torch.cuda.current_stream().wait_stream(s)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        rows, gx = step()
    moved = b.coords + 0.02 * torch.sin(torch.arange(b.coords.numel(), device="cuda", dtype=torch.float64)).reshape(x.shape)
    shift = torch.sin(40.0 * b.coords)                       # the same move for the same atom: sharing stays
    for new in (b.coords + 0.05 * shift, moved, b.coords):
        with torch.no_grad():
            x.copy_(torch.where(b.coords == 0, b.coords, new))
        graph.replay()
        torch.cuda.synchronize()
        r0, g0 = rows.clone(), gx.clone()
        r1, g1 = step()
        assert torch.equal(r0, r1) and torch.equal(g0, g1)


def test_drop_in_signal_leaves_the_callers_word_alone():
    """bad_ipot is the caller's, whatever it holds: it does not steer the call, and only a bad index is added to it."""
    from feffgpu_b200 import GPUPathStage, _lib
    P = phase("case_A014")
    st = GPUPathStage(P, device="cuda")
    nleg, B = 4, 700
    c, ip, _, _ = _list(P.nph, {nleg: B}, 6, seed=3)[0]
    c, ip = torch.tensor(c, device="cuda", dtype=st.rdtype), torch.tensor(ip, device="cuda")
    ref, rr = st.cchi(c, ip)
    bytes_ = int(st._lib.fg_cchi_workspace(st._h, B, nleg))
    assert bytes_ > 0
    for before in (0, 2, -1):
        word = torch.tensor([before], device="cuda", dtype=torch.int32)
        ws = torch.zeros(bytes_, dtype=torch.uint8, device="cuda")
        got, rf = torch.empty_like(ref), torch.empty_like(rr)
        _lib.check(st._lib.fg_cchi_ws(st._h, st.prec, B, nleg, c.data_ptr(), 0, ip.data_ptr(), got.data_ptr(),
                                      rf.data_ptr(), word.data_ptr(), ws.data_ptr(), bytes_,
                                      torch.cuda.current_stream().cuda_stream))
        assert torch.equal(got, ref) and torch.equal(rf, rr)
        assert int(word) == before


@pytest.mark.parametrize("dtype", DTYPES)
def test_workspace_on_an_8_byte_boundary(dtype):
    """Every call with a workspace of full size that starts 8 bytes past a 16-byte boundary: the one-kernel form's bits."""
    from feffgpu_b200 import GPUPathStage, PathBatch, _lib
    from feffgpu_b200.pad import resample_phase
    P = resample_phase(phase("cfg2_phase"), np.linspace(0.0, 20.0, 131))
    st = GPUPathStage(P, device="cuda", dtype=dtype)
    b = PathBatch(_list(P.nph, {2: 7, 4: 500}, 7, seed=4), nrows=3, device="cuda")
    q = torch.arange(1, 202, dtype=torch.float64, device="cuda") * 0.1
    S = st.linear_matrix(q.cpu().numpy()).double().contiguous()
    g = torch.randn(3, 201, dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(5))
    ref, cc, rf, offered = _rows(st, b, q, S, False)
    gref, _, _ = _grads(st, b, q, S, False, g, None)
    span, tspan, ps = st._span(S), st._span(S, True), st._paths_struct(b, b.coords, None)
    stream = torch.cuda.current_stream().cuda_stream

    def odd(n):
        return torch.empty(n + 8, dtype=torch.uint8, device="cuda")[8:]

    assert offered
    ws = odd(int(st._lib.fg_chi_reduce_workspace(st._h, C.byref(ps), 201)))
    rows = torch.empty_like(ref)
    _lib.check(st._lib.fg_chi_reduce(st._h, st.prec, C.byref(ps), 201, q.data_ptr(), S.data_ptr(), span.data_ptr(),
                                     rows.data_ptr(), None, None, ws.data_ptr(), ws.numel(), stream))
    ws = odd(int(st._lib.fg_chi_reduce_backward_workspace(st._h, C.byref(ps), 201)))
    gc = torch.empty_like(gref)
    _lib.check(st._lib.fg_chi_reduce_backward(st._h, st.prec, C.byref(ps), 201, q.data_ptr(), S.data_ptr(),
                                              span.data_ptr(), tspan.data_ptr(), g.data_ptr(), cc.data_ptr(),
                                              rf.data_ptr(), gc.data_ptr(), None, ws.data_ptr(), ws.numel(), stream))
    assert ws.data_ptr() % 16 == 8 and torch.equal(rows, ref) and torch.equal(gc, gref)
    sel = (b.nleg == 4).nonzero().squeeze(1)
    c, ip = b.coords[sel, :4].to(st.rdtype).contiguous(), b.ipots[sel, :4].contiguous()
    n = len(sel)
    ws, sig, reff = odd(int(st._lib.fg_cchi_workspace(st._h, n, 4))), *map(torch.empty_like, st.cchi(c, ip))
    _lib.check(st._lib.fg_cchi_ws(st._h, st.prec, n, 4, c.data_ptr(), int(dtype == torch.complex128), ip.data_ptr(),
                                  sig.data_ptr(), reff.data_ptr(), None, ws.data_ptr(), ws.numel(), stream))
    assert torch.equal(sig, st.cchi(c, ip)[0])
    gs = torch.randn(n, st.E, 2, dtype=st.rdtype, device="cuda", generator=torch.Generator("cuda").manual_seed(6))
    ws, x, y = odd(int(st._lib.fg_cchi_backward_workspace(st._h, n, 4))), torch.empty_like(c), torch.empty_like(c)
    for out, w, size in ((x, ws, ws.numel()), (y, torch.empty(256, dtype=torch.uint8, device="cuda"), 256)):
        _lib.check(st._lib.fg_cchi_backward(st._h, st.prec, n, 4, c.data_ptr(), int(dtype == torch.complex128),
                                            ip.data_ptr(), gs.data_ptr(), None, out.data_ptr(), w.data_ptr(), size, stream))
    assert torch.equal(x, y)


@pytest.mark.parametrize("backward", [False, True])
@pytest.mark.parametrize("case,counts", [("cfg4_fe_phase", {3: 33000}), ("case_A014", {4: (1 << 18) + 5})],
                         ids=["staged", "shared"])
def test_kernel_timing_spans_every_sub_batch(case, counts, backward):
    """A list one sub-batch and a little more: the time is of all of it, most of what the call takes on the device (the
    rest are the check, the sums' clearing and reading out, and in the backward the fine grid's adjoint)."""
    from feffgpu_b200 import GPUPathStage, PathBatch, _lib
    if backward and 3 in counts:
        pytest.skip("the staged form has no backward")
    st = GPUPathStage(phase(case), device="cuda")
    b = PathBatch(_list(st.P.nph, counts, 7, seed=9), nrows=3, device="cuda")
    q = torch.arange(1, 21, dtype=torch.float64, device="cuda")
    S = st.linear_matrix(q.cpu().numpy()).double().contiguous()
    g = torch.ones(3, 20, dtype=torch.float64, device="cuda")
    _, cc, rf = st._chi_reduce_forward(b, b.coords, None, q, S, st.prec, True)

    def call():
        if backward:
            st._chi_reduce_backward(b, b.coords, None, q, S, st.prec, g, cc, rf, False)
        else:
            st._chi_reduce_forward(b, b.coords, None, q, S, st.prec, False)

    call()
    e0, e1, ms = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True), C.c_float()
    st._lib.fg_set_kernel_timing(1)
    try:
        e0.record()
        call()
        e1.record()
        e1.synchronize()
        _lib.check(st._lib.fg_kernel_time_ms(C.byref(ms)))
    finally:
        st._lib.fg_set_kernel_timing(0)
    assert 0.5 * e0.elapsed_time(e1) <= ms.value <= e0.elapsed_time(e1)


def _own(nph, counts, seed):
    """Lists of paths with no two scatterers alike (every path has its own 0.05 A displacements)."""
    rng = np.random.default_rng(seed)
    return [(c + np.where(np.arange(c.shape[1])[None, :, None] > 0, rng.normal(0, 0.05, c.shape), 0.0), i, d, r)
            for c, i, d, r in _list(nph, counts, 6, seed=seed)]


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("case,nk", [("cfg2_phase", 131), ("case_A014", 0)])
@pytest.mark.parametrize("rest", [3, 1700], ids=["one part", "two parts"])
def test_list_without_sharing_in_every_call(dtype, case, nk, rest):
    """Two scatterers a class or more are not there: the forward goes on in the staged form, in as many parts as its tables
    fit the matrices' memory; the backward in the one-kernel form.  The bits of a call without workspace either way."""
    from feffgpu_b200 import GPUPathStage, PathBatch, _lib
    from feffgpu_b200.pad import resample_phase
    P = resample_phase(phase(case), np.linspace(0.0, 20.0, nk)) if nk else phase(case)
    st = GPUPathStage(P, device="cuda", dtype=dtype)
    real = 4 if dtype == torch.complex64 else 8
    entries = 16 if st.ilinit == 1 else 28                       # of a table's row, K edge and others
    cap = (1 << 30) // (8 * (st.L1 + 1) * entries * real)        # nine-leg paths whose tables fit 1 GiB
    counts = {4: 17000, 2: rest} if rest == 3 else {9: cap + rest}
    b = PathBatch(_own(P.nph, counts, 11), nrows=3, device="cuda")
    q = torch.arange(1, 31, dtype=torch.float64, device="cuda") * 0.5
    S = st.linear_matrix(q.cpu().numpy()).double().contiguous()
    got, cc, rf, offered = _rows(st, b, q, S, True)
    ref, cr, rr, _ = _rows(st, b, q, S, False)
    assert offered and torch.isfinite(torch.view_as_real(cr)).all()
    assert torch.equal(cc, cr) and torch.equal(got, ref) and torch.equal(rf, rr)
    if rest == 3:
        g = torch.randn(3, 30, dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(5))
        a, _, full = _grads(st, b, q, S, True, g, None)
        assert full and torch.equal(a, _grads(st, b, q, S, False, g, None)[0])
        sel = (b.nleg == 4).nonzero().squeeze(1)
        c, ip = b.coords[sel, :4].to(st.rdtype).contiguous(), b.ipots[sel, :4].contiguous()
        sig, reff = st.cchi(c, ip)
        x, y = torch.empty_like(sig), torch.empty_like(reff)
        _lib.check(st._lib.fg_cchi(st._h, st.prec, len(sel), 4, c.data_ptr(), int(real == 8), ip.data_ptr(), x.data_ptr(),
                                   y.data_ptr(), None, torch.cuda.current_stream().cuda_stream))
        assert int(st._lib.fg_cchi_workspace(st._h, len(sel), 4)) > 0 and torch.equal(sig, x) and torch.equal(reff, y)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("case,counts", [("cfg2_phase", {6: 900, 4: 300, 2: 9}), ("cfg4_fe_phase", {3: 3000})],
                         ids=["classes", "staged"])
def test_scratch_of_one_precision(dtype, case, counts, monkeypatch):
    """The stage's calls take scratch for their own precision, which is enough for the form; on a device without room for
    it they run with the least, and give the same rows (and the one-kernel form's gradients)."""
    from feffgpu_b200 import GPUPathStage, PathBatch, _lib
    from feffgpu_b200.pad import resample_phase
    P = phase(case) if 3 in counts else resample_phase(phase(case), np.linspace(0.0, 20.0, 131))
    st = GPUPathStage(P, device="cuda", dtype=dtype)
    b = PathBatch(_list(st.P.nph, counts, 7, seed=12), nrows=3, device="cuda")
    q = torch.arange(1, 102, dtype=torch.float64, device="cuda") * 0.15
    S = st.linear_matrix(q.cpu().numpy()).double().contiguous()
    g = torch.randn(3, 101, dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(3))
    lib, ps = st._lib, st._paths_struct(b, b.coords, None)
    for back in (0, 1):
        own, other = (int(lib.fg_share_workspace(st._h, p, b.n, b.nleg_max, 0 if back else 101, back))
                      for p in (st.prec, _lib.FG_FP64 if st.prec == _lib.FG_MIXED else _lib.FG_MIXED))
        call = lib.fg_chi_reduce_backward_workspace if back else lib.fg_chi_reduce_workspace
        least = 256 + (16 * 3 * 101 + 255) // 256 * 256
        if back:
            least = 256 + sum((v + 255) // 256 * 256 for v in (b.n * st.E * 16, b.n * 8, b.n * 256))
        assert int(call(st._h, C.byref(ps), 101)) == least + max(own, other)
    assert int(lib.fg_share_workspace(st._h, st.prec, b.n, b.nleg_max, 101, 0)) > 0
    sizes, empty = [], torch.empty

    def recorded(*args, **kw):
        if kw.get("dtype") == torch.uint8:
            sizes.append(args[0])
        return empty(*args, **kw)

    def full(*args, **kw):
        if kw.get("dtype") == torch.uint8 and args[0] == max(sizes):
            raise torch.cuda.OutOfMemoryError("full")
        return recorded(*args, **kw)

    def step():
        x = b.coords.clone().requires_grad_(True)
        rows = st.chi_reduce(b, q, S, coords=x)
        return rows.detach(), torch.autograd.grad(rows, x, g)[0]

    monkeypatch.setattr(torch, "empty", recorded)
    rows, gx = step()
    assert len(sizes) == 2
    one = st._chi_reduce_forward(b, b.coords, None, q, S, st.prec, True, one_kernel=True)
    gone = st._chi_reduce_backward(b, b.coords, None, q, S, st.prec, g, one[1], one[2], False, one_kernel=True)[0]
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as p:
        step()
        torch.cuda.synchronize()
    names = " ".join(e.key for e in p.key_averages())
    assert ("k_share_chain" if 6 in counts else "k_stage_energies") in names and "k_fused" not in names
    del sizes[:]
    sizes.append(256 + (16 * 3 * 101 + 255) // 256 * 256 + int(lib.fg_share_workspace(st._h, st.prec, b.n, b.nleg_max, 101, 0)))
    monkeypatch.setattr(torch, "empty", full)
    small, _ = step()
    assert torch.equal(small, rows) and torch.equal(rows, one[0])
    _same(gx, gone, {torch.complex64: 1e-5, torch.complex128: 1e-11}[dtype])
