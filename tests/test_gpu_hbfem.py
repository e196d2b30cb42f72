"""Harmonic-balance assembly on the GPU against the oracle restatement (which is itself
pinned to the reference gateway on linear materials, tests/test_oracle.py)."""
import numpy as np
import pytest
import torch
from conftest import bits_equal

from magpackage_b200 import material, quadrature, synth
from magpackage_b200.hbfem import AFT, assemble_hbfem
from magpackage_b200.plan import AssemblyPlan
from oracle.oracle import mex_inputs

pytestmark = pytest.mark.gpu


def _case(port, harmonics, n=(5, 4, 3), seed=12, scale=1.0, imag=True):
    mesh = synth.kuhn_box(*n, seed=seed)
    tags = synth.cube_layout(mesh)
    edges, t2e, sign = port.generate_edges(mesh.T)
    E = edges.shape[0]
    m = mex_inputs(mesh.P, mesh.T, t2e, sign, tags)
    pk = material.pack_material_data(synth.standard_materials())
    plan = AssemblyPlan(mesh.P, mesh.T, t2e, E, tags, sign)
    plan.set_materials(pk)
    rng = np.random.default_rng(seed)
    K = len(harmonics)
    # a spread of magnitudes drives the iron through the spline's interior, knee and extrapolation
    amp = scale * np.exp(rng.uniform(-4, 1, (E, K)))
    sol = amp * rng.normal(0, 1, (E, K)) + (1j * amp * rng.normal(0, 1, (E, K)) if imag else 0.0)
    return plan, m, pk, sol, E


@pytest.mark.parametrize("harmonics,imag", [((0, 1, 3), True), ((1, 3, 5, 7), True), ((0, 1), False), ((1,), True),
                                            ((1, 3, 5, 7, 9), True)])
def test_hbfem_matches_oracle(oracle_port, harmonics, imag):
    plan, m, pk, sol, E = _case(oracle_port, harmonics, imag=imag)
    aft = AFT(harmonics)
    qw, val, curl = quadrature.reference_data(2)
    K = len(harmonics)
    I, J, V, Rr, Rc, Rre, Rim = oracle_port.hbfem(m, sol, aft.D, aft.P, qw, curl, pk, True)
    R, vals = assemble_hbfem(plan, sol, aft, True)
    R = R.cpu().numpy()
    # residual: sparse(R_rows, R_cols, R_val, Ndof, K), summed in order of appearance
    lin = Rr + (Rc - 1) * E
    ref_re = oracle_port.sparse_vec(lin, Rre, E * K).reshape(K, E)
    ref_im = oracle_port.sparse_vec(lin, Rim, E * K).reshape(K, E)
    assert bits_equal(np.real(R), ref_re)
    assert bits_equal(np.imag(R), ref_im)
    assert np.abs(ref_re).max() > 0 and np.abs(ref_im).max() > 0
    # Jacobian: the first harmonic's block (scaling 1) on the structural pattern
    first = I <= E
    rp, ci, rv = oracle_port.sparse_csr(I[first], J[first], V[first], E, drop_zeros=False)
    assert np.array_equal(plan.row_ptr.cpu().numpy(), rp)
    assert np.array_equal(plan.col_idx.cpu().numpy(), ci)
    assert bits_equal(vals.cpu().numpy(), rv)


def test_hbfem_residual_only_and_errors(oracle_port):
    plan, m, pk, sol, E = _case(oracle_port, (1, 3))
    aft = AFT((1, 3))
    R1, v1 = assemble_hbfem(plan, sol, aft, True)
    R0, v0 = assemble_hbfem(plan, sol, aft, False)
    assert v0 is None and torch.equal(R0, R1)
    from magpackage_b200 import _lib
    with pytest.raises(_lib.MagError):
        assemble_hbfem(plan, np.zeros((E, 17)), AFT(list(range(17))), False)  # more than 16 harmonics


def test_hbfem_device_resident_field_gives_the_same_bits(oracle_port):
    """A complex CUDA tensor or a (re, im) pair already in [K, Ndof] layout is used without
    a host round trip and gives the host array's result."""
    plan, m, pk, sol, E = _case(oracle_port, (0, 1, 3))
    aft = AFT((0, 1, 3))
    R0, v0 = assemble_hbfem(plan, sol, aft, True)
    R1, v1 = assemble_hbfem(plan, torch.as_tensor(sol, device="cuda"), aft, True)
    pair = (torch.as_tensor(np.ascontiguousarray(sol.real.T), device="cuda"),
            torch.as_tensor(np.ascontiguousarray(sol.imag.T), device="cuda"))
    R2, v2 = assemble_hbfem(plan, pair, aft, True)
    for R, v in ((R1, v1), (R2, v2)):
        assert torch.equal(R, R0) and torch.equal(v, v0)
    with pytest.raises(ValueError):
        assemble_hbfem(plan, pair[0][:2], aft, False)


@pytest.mark.parametrize("harmonics,samples,weights,schedule", [
    ((0, 1), 5, "equal", None),            # fewer samples than warps
    ((1, 3), 16, "equal", None),           # the 16-sample form filled
    ((1, 3), 17, "equal", "two_pass"),     # 24-sample form, padded; DC block through the row reduction
    ((0, 1, 2, 5), 24, "equal", None),
    ((1, 15), 31, "equal", None),
    ((1, 3, 5), 33, "equal", None),        # more samples than the register forms hold
    (tuple(range(16)), 64, "equal", None),  # most harmonics
    (tuple(range(16)), 128, "equal", "two_pass"),
    ((1, 3), 32, "uneven", None),          # general kernel
])
def test_hbfem_sample_counts_and_weights(oracle_port, harmonics, samples, weights, schedule):
    """Every form of the element kernel against the oracle, 354 elements (a ragged last CTA)."""
    from magpackage_b200 import _lib

    plan, m, pk, sol, E = _case(oracle_port, harmonics, n=(1, 1, 59), seed=3)
    aft = AFT(harmonics, n_time_steps=samples)
    assert aft.num_time_steps == samples
    qw, val, curl = quadrature.reference_data(2)
    if weights == "uneven":
        qw = qw * np.array([1.0, 0.5, 1.25, 1.25])
        plan.set_quadrature(qw, curl, val)
    if schedule == "two_pass":
        plan.set_schedule(_lib.SCHEDULE_TWO_PASS)
    K = len(harmonics)
    I, J, V, Rr, Rc, Rre, Rim = oracle_port.hbfem(m, sol, aft.D, aft.P, qw, curl, pk, True)
    R, vals = assemble_hbfem(plan, sol, aft, True)
    R = R.cpu().numpy()
    lin = Rr + (Rc - 1) * E
    assert bits_equal(np.real(R), oracle_port.sparse_vec(lin, Rre, E * K).reshape(K, E))
    assert bits_equal(np.imag(R), oracle_port.sparse_vec(lin, Rim, E * K).reshape(K, E))
    first = I <= E
    _, _, rv = oracle_port.sparse_csr(I[first], J[first], V[first], E, drop_zeros=False)
    assert bits_equal(vals.cpu().numpy(), rv)


@pytest.mark.parametrize("harmonics,samples,weights,n", [
    ((1,), 256, "equal", (1, 1, 59)),            # more samples than the constant-curl kernel's shared memory
    ((1, 3), 256, "equal", (1, 1, 59)),          # holds: the general kernel compiled for 1 to 4 harmonics
    ((1, 3, 5), 256, "equal", (1, 1, 59)),
    ((0, 1, 3, 5), 256, "equal", (1, 1, 59)),
    ((1, 3, 5, 7, 9), 256, "equal", (1, 1, 59)),  # and with the count at run time
    ((1,), 32, "uneven", (1, 1, 59)),
    ((1, 3, 5), 32, "uneven", (1, 1, 59)),
    ((0, 1, 3, 5), 17, "uneven", (1, 1, 59)),
    ((1,), 33, "equal", (22, 22, 21)),           # one harmonic on 60,984 elements: general kernel
])
def test_hbfem_general_kernel(oracle_port, harmonics, samples, weights, n):
    """The general element kernel against the oracle, with and without the DC block."""
    plan, m, pk, sol, E = _case(oracle_port, harmonics, n=n, seed=4)
    aft = AFT(harmonics, n_time_steps=samples)
    assert aft.num_time_steps == samples
    qw, val, curl = quadrature.reference_data(2)
    if weights == "uneven":
        qw = qw * np.array([1.0, 0.5, 1.25, 1.25])
        plan.set_quadrature(qw, curl, val)
    K = len(harmonics)
    I, J, V, Rr, Rc, Rre, Rim = oracle_port.hbfem(m, sol, aft.D, aft.P, qw, curl, pk, True)
    R, vals = assemble_hbfem(plan, sol, aft, True)
    assert torch.equal(assemble_hbfem(plan, sol, aft, False)[0], R)
    R = R.cpu().numpy()
    lin = Rr + (Rc - 1) * E
    assert bits_equal(np.real(R), oracle_port.sparse_vec(lin, Rre, E * K).reshape(K, E))
    assert bits_equal(np.imag(R), oracle_port.sparse_vec(lin, Rim, E * K).reshape(K, E))
    first = I <= E
    _, _, rv = oracle_port.sparse_csr(I[first], J[first], V[first], E, drop_zeros=False)
    assert bits_equal(vals.cpu().numpy(), rv)


def test_hbfem_both_kernels_give_the_same_bits(oracle_port):
    """Two harmonics on 196,608 elements: a residual alone takes the general kernel, one with the DC
    block the constant-curl kernel."""
    plan, m, pk, sol, E = _case(oracle_port, (1, 3), n=(32, 32, 32), seed=5)
    aft = AFT((1, 3), n_time_steps=33)
    assert torch.equal(assemble_hbfem(plan, sol, aft, False)[0], assemble_hbfem(plan, sol, aft, True)[0])


@pytest.mark.parametrize("samples", [9, 20, 32, 40, 256])
def test_hbfem_real_transform_of_an_infinite_field(oracle_port, samples):
    """Without Im P the imaginary residual is zero, also where a field value is infinite and its
    samples are infinities and NaN; entries the value does not reach keep the finite field's bits."""
    import ctypes as C

    from magpackage_b200 import _lib

    harmonics = (0, 1, 2)
    plan, m, pk, sol, E = _case(oracle_port, harmonics, n=(3, 2, 3), seed=6)
    dr, di, pr, _ = AFT(harmonics, n_time_steps=samples).device_operators()
    K, res = len(harmonics), []
    for bad in (False, True):
        sr = torch.as_tensor(np.ascontiguousarray(sol.real.T), device="cuda")
        si = torch.as_tensor(np.ascontiguousarray(sol.imag.T), device="cuda")
        if bad:
            sr[1, 5] = float("inf")
        re, im = torch.full_like(sr, 7.0), torch.full_like(sr, 7.0)
        p = lambda t: C.c_void_p(t.data_ptr())
        _lib.check(_lib.lib().mag_assemble_hbfem(plan._h, p(sr), p(si), K, p(dr), p(di), p(pr), None, samples, None,
                                                 p(re), p(im), _lib.stream_ptr()))
        assert torch.count_nonzero(im) == 0
        res.append(re)
    bad = ~torch.isfinite(res[1])
    assert 0 < int(bad[0].sum()) < E
    assert torch.equal(res[0][~bad], res[1][~bad])


def test_hbfem_workspace_is_bounded_and_reported():
    """A handle's pool keeps no more workspace than the handle's own arrays hold; the rest goes back at
    the next synchronisation, and what it keeps counts in device_bytes. Up to three harmonics on a
    large mesh need no workspace at all."""
    import ctypes as C

    from magpackage_b200 import _lib
    from magpackage_b200.plan import generate_edges

    def held(plan):
        torch.cuda.synchronize()
        info = _lib.MeshInfo()
        _lib.check(_lib.lib().mag_mesh_get_info(plan._h, C.byref(info)))
        return int(info.device_bytes)

    mesh = synth.kuhn_box(54, seed=2)  # 944,784 elements: 96 bytes an element and harmonic
    edges, t2e, sign = generate_edges(mesh.T)
    plan = AssemblyPlan(mesh.P, mesh.T, t2e, edges.shape[0], synth.cube_layout(mesh), sign)
    plan.set_materials(material.pack_material_data(synth.standard_materials()))
    small, base = 256 << 20, held(plan)
    assert base > small
    for K, calc_j in ((3, True), (3, False), (1, True), (6, False), (16, False)):
        aft = AFT(tuple(range(K)), n_time_steps=33)
        need = plan.num_elements * 96 * K
        g = torch.Generator(device="cuda").manual_seed(K)
        sol = tuple(1e-3 * torch.randn((K, plan.num_dofs), dtype=torch.float64, device="cuda", generator=g) for _ in range(2))
        aft.device_operators()
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        free0 = torch.cuda.mem_get_info()[0] + torch.cuda.memory_reserved()
        R, _ = assemble_hbfem(plan, sol, aft, calc_j)
        torch.cuda.synchronize()
        free1 = torch.cuda.mem_get_info()[0] + torch.cuda.memory_reserved()
        grown = held(plan) - base
        assert free0 - free1 <= base + (64 << 20), (K, free0 - free1)  # (64 MB: kernels loaded at their first launch)
        assert grown <= base + (32 << 20), (K, grown)                  # (32 MB: granularity of the pool)
        if K == 3:
            assert need > small and grown == 0
        if K == 1:
            assert need < small and grown >= need
        if K == 16:
            assert need > base + (64 << 20)
        del R, sol
    plan.close()


@pytest.mark.parametrize("harmonics,samples", [((1,), 33), ((1, 3), 40), ((1,), 7), ((1,), 20), ((0, 1), 8), ((1, 3), 16),
                                               ((0, 1, 2), 33)])
def test_hbfem_one_quadrature_point(oracle_port, harmonics, samples):
    """One point on 47,880 elements, where either kernel may serve: with the DC block and alone."""
    plan, m, pk, sol, E = _case(oracle_port, harmonics, n=(21, 20, 19), seed=7)
    aft = AFT(harmonics, n_time_steps=samples)
    assert aft.num_time_steps == samples
    qw, val, curl = quadrature.reference_data(1)
    plan.set_quadrature(qw, curl, val)
    K = len(harmonics)
    I, J, V, Rr, Rc, Rre, Rim = oracle_port.hbfem(m, sol, aft.D, aft.P, qw, curl, pk, True)
    lin = Rr + (Rc - 1) * E
    want_re = oracle_port.sparse_vec(lin, Rre, E * K).reshape(K, E)
    want_im = oracle_port.sparse_vec(lin, Rim, E * K).reshape(K, E)
    first = I <= E
    _, _, rv = oracle_port.sparse_csr(I[first], J[first], V[first], E, drop_zeros=False)
    for calc_j in (True, False):
        R, vals = assemble_hbfem(plan, sol, aft, calc_j)
        R = R.cpu().numpy()
        assert bits_equal(np.real(R), want_re) and bits_equal(np.imag(R), want_im)
        assert vals is None or bits_equal(vals.cpu().numpy(), rv)
