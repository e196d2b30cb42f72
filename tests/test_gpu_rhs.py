"""Right-hand-side kernels on the GPU against the oracle, bit for bit: the winding vector
(assemble_winding_kernel_mex.cpp) and the source vector (assemble_source_kernel_mex.cpp),
through the MEX-compatible entry points (golden fixtures of the reference) and the mesh
handle (sparse(I(valid), 1, V(valid), Ndof, 1) of the oracle's pairs)."""
import numpy as np
import pytest
import torch
from conftest import bits_equal, load_golden

from magpackage_b200 import _lib, quadrature, synth
from magpackage_b200.assembler import Assembler, DofHandler, Mesh, Winding
from magpackage_b200.plan import AssemblyPlan, generate_edges
from oracle.oracle import mex_inputs

pytestmark = pytest.mark.gpu


def _mex_winding(L, m, coil, field, udir, scale, qw, val):
    p = _lib.dptr
    ne = m.ne
    I, V = np.zeros(6 * ne), np.zeros(6 * ne)
    f = None if field is None else np.ascontiguousarray(field, dtype=np.float64)
    u = np.ascontiguousarray(udir, dtype=np.float64)
    _lib.check(L.mag_mex_winding(p(m.P), m.nn, p(m.T), ne, p(m.Dofs), p(m.Signs), p(m.Tags), float(coil), p(f),
                                 p(u), float(scale), p(qw), qw.size, p(val), p(I), p(V)))
    return I, V


@pytest.mark.parametrize("name", ["one_hex", "cube3"])
def test_mex_winding_and_source_match_golden(name):
    d = load_golden(name)
    L = _lib.lib()
    m = mex_inputs(d["P"], d["T0"], d["t2e"], d["sign"], d["tags"])
    qw, val = np.ascontiguousarray(d["qw"]), np.ascontiguousarray(d["val"])
    for field, key in ((None, "u"), (d["win_field"], "f")):
        I, V = _mex_winding(L, m, d["win_coil"], field, d["win_dir"], d["win_scale"], qw, val)
        assert bits_equal(I, d[f"win_{key}_I"]) and bits_equal(V, d[f"win_{key}_V"])
    js = np.ascontiguousarray(d["src_js"])
    I, V = np.zeros(6 * m.ne), np.zeros(6 * m.ne)
    p = _lib.dptr
    _lib.check(L.mag_mex_source(p(m.P), m.nn, p(m.T), m.ne, p(m.Dofs), p(m.Signs), p(js), p(qw), qw.size, p(val),
                                p(I), p(V)))
    assert bits_equal(I, d["src_I"]) and bits_equal(V, d["src_V"])


def test_mex_source_signs_of_zeros(oracle_port):
    """f * sign of an element without a source is a zero with the edge's sign, as in the reference's
    pairs (assemble_source_kernel_mex.cpp:46-114): signs of zeros included, every bit is the oracle's."""
    mesh = synth.kuhn_box(3, 2, 4, seed=8)
    edges, t2e, sign = oracle_port.generate_edges(mesh.T)
    sign = sign.copy()
    sign[::2] *= -1
    m = mex_inputs(mesh.P, mesh.T, t2e, sign, synth.cube_layout(mesh))
    qw, val, curl = quadrature.reference_data(2)
    js = np.random.default_rng(8).normal(size=(m.ne, 3))
    js[1::3] = 0.0
    js[2::3] = 1e-13  # below the reference's cut-off
    Io, Vo = oracle_port.source(m, js, qw, val)
    I, V = np.ones(6 * m.ne), np.ones(6 * m.ne)
    p = _lib.dptr
    _lib.check(_lib.lib().mag_mex_source(p(m.P), m.nn, p(m.T), m.ne, p(m.Dofs), p(m.Signs), p(js), p(qw), qw.size,
                                         p(val), p(I), p(V)))
    assert np.array_equal(I, Io)
    assert np.sum((Vo == 0) & np.signbit(Vo)) > 100
    assert np.array_equal(V.view(np.int64), Vo.view(np.int64))


def _vector(port, I, V, n):
    k = I > 0
    return port.sparse_vec(I[k], V[k], n)


@pytest.mark.parametrize("coil", [synth.IRON, synth.ALUMINIUM, 77])
def test_winding_vector_matches_oracle(oracle_port, coil):
    mesh = synth.kuhn_box(7, 6, 5, seed=21)
    tags = synth.cube_layout(mesh)
    edges, t2e, sign = oracle_port.generate_edges(mesh.T)
    E = edges.shape[0]
    dofs = t2e.copy()
    rng = np.random.default_rng(coil)
    dofs[rng.random(dofs.shape) < 0.05] = -1  # edges without an unknown
    m = mex_inputs(mesh.P, mesh.T, dofs, sign, tags)
    qw, val, curl = quadrature.reference_data(2)
    plan = AssemblyPlan(mesh.P, mesh.T, dofs, E, tags, sign)
    field = rng.normal(size=(mesh.num_elements, 3))
    udir = np.array([0.2, 0.9, -0.4])
    for f in (None, field):
        I, V = oracle_port.winding(m, float(coil), f, udir, 3.3e5, qw, val)
        ref = _vector(oracle_port, I, V, E)
        got = plan.winding(coil, udir, 3.3e5, dir_field=None if f is None else torch.as_tensor(f, device="cuda"))
        assert bits_equal(got.cpu().numpy(), ref)
        assert (np.abs(ref).max() > 0) == (coil != 77)
        Ig, Vg = _mex_winding(_lib.lib(), m, coil, f, udir, 3.3e5, qw, val)
        assert bits_equal(Ig, I) and bits_equal(Vg, V)


def test_assembler_winding_surface(oracle_port):
    mesh_s = synth.kuhn_box(6, seed=2)
    tags = synth.cube_layout(mesh_s)
    mesh = Mesh(mesh_s.P, mesh_s.T, tags)
    dh = DofHandler(mesh)
    dh.distribute_dofs()
    asm = Assembler(mesh, dh)
    w1 = Winding.create("A", synth.IRON, 120, 0.5, 2e-3, (0, 0, 2.0))
    w2 = Winding.create("B", synth.ALUMINIUM, 40, 0.1, 1e-3, (1.0, 1.0, 0))
    assert np.allclose(np.linalg.norm(w1.Direction), 1.0) and np.allclose(np.linalg.norm(w2.Direction), 1.0)
    w2.set_direction_field(np.random.default_rng(1).normal(size=(mesh.num_elements, 3)))
    C = asm.assemble_winding([w1, w2])
    assert C.shape == (dh.NumGlobalDofs, 2)
    dofs, signs = (torch.as_tensor(a).cpu().numpy() for a in dh.pack_for_kernel())
    m = mex_inputs(mesh_s.P, mesh_s.T, dofs, signs, tags)
    qw, val, curl = quadrature.reference_data(2)
    for k, w in enumerate((w1, w2)):
        I, V = oracle_port.winding(m, float(w.RegionID), w.DirectionField, w.Direction, w.Turns / w.CrossSectionArea,
                                   qw, val)
        assert bits_equal(C[:, k].cpu().numpy(), _vector(oracle_port, I, V, dh.NumGlobalDofs))
    with pytest.raises(ValueError):
        w2.set_direction_field(np.zeros((3, 3)))
        asm.assemble_winding(w2)


@pytest.mark.parametrize("flip", [False, True])
def test_element_b_matches_postprocessor(oracle_port, flip):
    """mag_element_b against PostProcessor.computeElementB restated (PostProcessor.m:64-126):
    B per element within 1e-12 of its rounding scale (MATLAB's BLAS products have no fixed
    summation order, so this is a tolerance, not a bit comparison), |B|^2 = B.B bit for bit;
    with the mesh's own signs and with explicitly flipped ones."""
    from oracle.oracle import element_b
    from test_oracle import uniform_field_edges

    mesh = synth.kuhn_box(9, 7, 8, seed=5)
    tags = synth.cube_layout(mesh)
    edges, t2e, sign = oracle_port.generate_edges(mesh.T)
    if flip:
        sign = sign.copy()
        sign[::3] *= -1
    E = edges.shape[0]
    plan = AssemblyPlan(mesh.P, mesh.T, t2e, E, tags, sign)
    rng = np.random.default_rng(4)
    for sol in (rng.normal(0, 1e-2, E), uniform_field_edges(mesh.P, edges, np.array([0.2, 0.5, -1.1]))):
        b, bsq = plan.element_b(torch.as_tensor(sol, device="cuda"))
        b, bsq = b.cpu().numpy(), bsq.cpu().numpy()
        B, scale = element_b(mesh.P, mesh.T, t2e, sign, sol)
        assert np.all(np.abs(b - B) <= 1e-12 * scale + 1e-300)
        assert bits_equal(bsq, (b[:, 0] * b[:, 0] + b[:, 1] * b[:, 1]) + b[:, 2] * b[:, 2])
    plan.close()


@pytest.mark.parametrize("order", [1, 2])
@pytest.mark.parametrize("sigma", ["one", "none", "slab", "all"])
@pytest.mark.parametrize("n,absent", [((1, 1, 1), 0.0), ((9, 4, 5), 0.0), ((9, 8, 9), 0.05)])
def test_mass_and_source_match_oracle(oracle_port, n, absent, sigma, order):
    """M(sigma) through the tile blocks and the source vector: one element to several tiles, no,
    few or all conducting elements, dofs missing, one and four quadrature points."""
    mesh = synth.kuhn_box(*n, seed=5)
    tags = synth.cube_layout(mesh)
    edges, t2e, sign = oracle_port.generate_edges(mesh.T)
    E = edges.shape[0]
    rng = np.random.default_rng(n[0])
    dofs = t2e.copy()
    dofs[rng.random(dofs.shape) < absent] = -1
    m = mex_inputs(mesh.P, mesh.T, dofs, sign, tags)
    qw, val, curl = quadrature.reference_data(order)
    plan = AssemblyPlan(mesh.P, mesh.T, dofs, E, tags, sign)
    plan.set_quadrature(qw, curl, val)
    assert plan.info.schedule == _lib.SCHEDULE_TILE_BLOCKS
    s = rng.uniform(0.5, 2.0, mesh.num_elements) * synth.SIGMA_AL
    s = {"one": None, "none": 0.0 * s, "slab": np.where(tags == synth.ALUMINIUM, s, 1e-13), "all": s}[sigma]
    I, J, V = oracle_port.mass(m, np.ones(mesh.num_elements) if s is None else s, qw, val)
    keep = (I > 0) & (J > 0)
    _, _, ref = oracle_port.sparse_csr(I[keep], J[keep], V[keep], E, drop_zeros=False)
    got = plan.mass(None if s is None else torch.as_tensor(s, device="cuda"))
    assert bits_equal(got.cpu().numpy(), ref)
    js = rng.normal(size=(mesh.num_elements, 3)) * (rng.random(mesh.num_elements) < 0.7)[:, None]
    I, V = oracle_port.source(m, js, qw, val)
    assert bits_equal(plan.source(torch.as_tensor(js, device="cuda")).cpu().numpy(), _vector(oracle_port, I, V, E))
    plan.check()


@pytest.mark.parametrize("n,absent,weights", [((33, 32, 32), 0.0, "equal"), ((34, 33, 31), 0.03, "uneven"),
                                              ((33, 32, 32), 0.0, "captured")])
def test_residual_alone_equals_jacobian_call(n, absent, weights):
    """The residual-only path of larger meshes gives the Jacobian call's residual (which the other
    tests pin to the oracle) bit for bit, also with dofs missing, with uneven weights, and replayed
    from a graph."""
    from magpackage_b200.material import pack_material_data
    from magpackage_b200.plan import generate_edges

    mesh = synth.kuhn_box(*n, seed=2)
    assert mesh.num_elements >= 200000
    edges, t2e, sign = generate_edges(mesh.T)
    g = torch.Generator(device="cuda").manual_seed(1)
    dofs = torch.where(torch.rand(t2e.shape, generator=g, device="cuda") < absent, -1, t2e.long()).int()
    plan = AssemblyPlan(mesh.P, mesh.T, dofs, int(edges.shape[0]), synth.cube_layout(mesh), sign)
    plan.set_materials(pack_material_data(synth.standard_materials()))
    if weights == "uneven":
        qw, val, curl = quadrature.reference_data(2)
        plan.set_quadrature(qw * np.array([1.0, 0.5, 1.25, 1.25]), curl, val)
    sol = 3e-4 * torch.randn(plan.num_dofs, dtype=torch.float64, device="cuda", generator=g)
    _, want = plan.jacobian(sol)
    if weights == "captured":
        got = plan.new_vector()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            plan.jacobian(sol, None, got, calc_j=False)
        got.zero_()
        graph.replay()
    else:
        _, got = plan.jacobian(sol, calc_j=False)
    assert torch.equal(got, want) and float(want.abs().max()) > 0
    plan.check()


def test_residuals_of_one_mesh_from_several_threads():
    """Threads with a stream each evaluate residuals of their own states on one mesh handle; each
    gets its state's, bit for bit."""
    import threading

    from magpackage_b200.material import pack_material_data
    from magpackage_b200.plan import generate_edges

    mesh = synth.kuhn_box(33, seed=2)
    assert mesh.num_elements >= 200000
    edges, t2e, sign = generate_edges(mesh.T)
    plan = AssemblyPlan(mesh.P, mesh.T, t2e, int(edges.shape[0]), synth.cube_layout(mesh), sign)
    plan.set_materials(pack_material_data(synth.standard_materials()))
    g = torch.Generator(device="cuda").manual_seed(1)
    sols = [3e-4 * torch.randn(plan.num_dofs, dtype=torch.float64, device="cuda", generator=g) for _ in range(4)]
    want = [plan.jacobian(x)[1] for x in sols]
    got = [[plan.new_vector() for _ in range(24)] for _ in sols]
    torch.cuda.synchronize()

    def work(x, outs):
        with torch.cuda.stream(torch.cuda.Stream()):
            for r in outs:
                plan.jacobian(x, None, r, calc_j=False)
            torch.cuda.current_stream().synchronize()

    threads = [threading.Thread(target=work, args=a) for a in zip(sols, got)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for w, outs in zip(want, got):
        assert all(torch.equal(w, r) for r in outs)
    plan.check()


@pytest.mark.parametrize("beside", ["source", "two_pass"])
def test_sources_of_one_mesh_from_several_threads(beside):
    """Threads with a stream each assemble source vectors of their own densities on one mesh handle,
    or sources beside two-pass mass matrices (which use the same scratch); each gets its own result,
    bit for bit."""
    import threading

    from magpackage_b200.plan import generate_edges

    mesh = synth.kuhn_box(33, seed=2)
    edges, t2e, sign = generate_edges(mesh.T)
    plan = AssemblyPlan(mesh.P, mesh.T, t2e, int(edges.shape[0]), synth.cube_layout(mesh), sign)
    g = torch.Generator(device="cuda").manual_seed(1)
    js = [torch.randn((mesh.num_elements, 3), dtype=torch.float64, device="cuda", generator=g) for _ in range(4)]
    calls = [lambda out, j=j: plan.source(j, out) for j in js]
    outs = [[plan.new_vector() for _ in range(24)] for _ in js]
    if beside == "two_pass":
        plan.set_schedule(_lib.SCHEDULE_TWO_PASS)
        for k in (1, 3):
            calls[k] = lambda out, s=js[k][:, 0].abs().contiguous(): plan.mass(s, out)
            outs[k] = [plan.new_values() for _ in range(24)]
    want = [f(torch.empty_like(o[0])) for f, o in zip(calls, outs)]
    torch.cuda.synchronize()

    def work(f, mine):
        with torch.cuda.stream(torch.cuda.Stream()):
            for r in mine:
                f(r)
            torch.cuda.current_stream().synchronize()

    threads = [threading.Thread(target=work, args=a) for a in zip(calls, outs)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for w, mine in zip(want, outs):
        assert float(w.abs().max()) > 0 and all(torch.equal(w, r) for r in mine)
    plan.check()


def test_residual_needs_no_memory_of_its_own():
    """From 200,000 elements on a residual alone goes through element entries: they lie in the handle's
    element scratch, so that a mesh above that size holds no more bytes an element than one below (an
    own buffer was 48; the two meshes' rows per element differ by 1 %)."""
    held = []
    for n in (32, 34):
        mesh = synth.kuhn_box(n, seed=2)
        edges, t2e, sign = generate_edges(mesh.T)
        plan = AssemblyPlan(mesh.P, mesh.T, t2e, edges.shape[0], synth.cube_layout(mesh), sign)
        held.append(plan.info.device_bytes / plan.num_elements)
        assert (plan.num_elements >= 200000) == (n == 34)
        plan.close()
    assert abs(held[1] - held[0]) < 16, held


def test_residuals_beside_sources_of_one_mesh():
    """Residuals on one stream and sources on another, in turn from one thread, share the handle's
    scratch: every result is the same bits as alone."""
    from magpackage_b200.material import pack_material_data

    mesh = synth.kuhn_box(33, seed=2)
    edges, t2e, sign = generate_edges(mesh.T)
    plan = AssemblyPlan(mesh.P, mesh.T, t2e, int(edges.shape[0]), synth.cube_layout(mesh), sign)
    plan.set_materials(pack_material_data(synth.standard_materials()))
    g = torch.Generator(device="cuda").manual_seed(3)
    sol = 3e-4 * torch.randn(plan.num_dofs, dtype=torch.float64, device="cuda", generator=g)
    js = torch.randn((mesh.num_elements, 3), dtype=torch.float64, device="cuda", generator=g)
    want_r, want_s = plan.jacobian(sol, calc_j=False)[1], plan.source(js)
    rs, ss = ([plan.new_vector() for _ in range(24)] for _ in range(2))
    s1, s2 = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    for r, v in zip(rs, ss):
        plan.jacobian(sol, None, r, calc_j=False, stream=s1)
        plan.source(js, v, stream=s2)
    torch.cuda.synchronize()
    assert float(want_r.abs().max()) > 0 and float(want_s.abs().max()) > 0
    assert all(torch.equal(want_r, r) for r in rs) and all(torch.equal(want_s, v) for v in ss)
    plan.check()
