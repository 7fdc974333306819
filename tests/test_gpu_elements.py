"""K2 parity: fused element kernels + deterministic CSR gather vs the CPU oracle, every kind.

Reference: ElementSolid::{update_secondary_values, calc_f_int, calc_jacobian}
(src/fem/element_solid.rs:124-224), Elements loops (src/fem/elements.rs:132-205), COO assembly
(src/base/assembly.rs:38-139).  Tolerance: relative (normwise) 1e-12; CSR bit-reproducible.
"""
import numpy as np
import pytest

import oracle
from gpu_util import assert_close, perturbed_mesh, plastic_ddu
from pmsim_b200 import mesh as M

pytestmark = pytest.mark.gpu

E, NU, H, Z0 = 2e5, 0.3, 1e3, 250.0
KINDS = [M.TRI3, M.TRI6, M.QUA4, M.QUA8, M.QUA9, M.TET4, M.HEX8, M.HEX20, M.TRI10, M.TRI15]
GRID = {2: (4, 3, 1), 3: (2, 2, 2)}


def make(kind, model=1, ngauss=0, seed=0):
    from pmsim_b200.elements import Elements, Material
    m = perturbed_mesh(kind, seed=seed, n=GRID[M.KIND_NDIM[kind]])
    mat = Material.von_mises(E, NU, H, Z0) if model == 1 else Material.linear_elastic(E, NU)
    g = Elements(m, mat, ngauss=ngauss)
    o = oracle.OracleElements(m, model, oracle.Params(E, NU, H, Z0), ngauss=ngauss, sym_tol=-1.0)
    return m, g, o


def oracle_csr_values(o, indptr, indices):
    ip, ix, data = o.assemble_kk_csr()
    assert np.array_equal(ip, indptr) and np.array_equal(ix, indices)
    return data


@pytest.mark.parametrize("kind", KINDS, ids=[M.KIND_NAMES[k] for k in KINDS])
def test_fused_update_and_assemble_matches_oracle(kind):
    m, g, o = make(kind)
    indptr, indices = g.csr_pattern()
    g.initialize_internal_values()
    o.initialize()
    # iteration 0 of a step: assemble from the initial (elastic) state
    assert np.all(g.assemble_f_int() == 0.0)
    k0 = g.assemble_kk()
    assert_close(k0, oracle_csr_values(o, indptr, indices), what="K elastic")
    # one Newton update from the backed-up state, then F_int and K on the updated state
    ddu = plastic_ddu(m, seed=kind)
    g.backup_secondary_values()
    ff = np.zeros(g.ndof)
    kv = np.zeros(g.nnz)
    g.update_and_assemble(ddu, ff, kv)
    o.update_secondary_values(ddu)
    sig, ivs, el = g.get_state()
    assert np.array_equal(el, o.elastic), "elastic flags differ"
    assert 0 < (1 - el.mean()) < 1, "expected a mix of elastic and plastic IPs"
    assert_close(sig, o.sig, what="sigma")
    assert_close(ivs, o.ivs, what="[z, lambda]")
    assert_close(ff, o.assemble_f_int(), what="f_int")
    assert_close(kv, oracle_csr_values(o, indptr, indices), what="K")


@pytest.mark.parametrize("kind", [M.QUA8, M.HEX20], ids=["qua8", "hex20"])
def test_separate_calls_match_fused(kind):
    """update_secondary + assemble_f_int + assemble_kk == fused call (to rounding: the two kernel
    instantiations may fuse multiply-adds differently)."""
    m, g, o = make(kind, seed=3)
    ddu = plastic_ddu(m, seed=5)
    g.initialize_internal_values()
    g.backup_secondary_values()
    ff1, kv1 = np.zeros(g.ndof), np.zeros(g.nnz)
    g.update_and_assemble(ddu, ff1, kv1)
    s1 = g.get_state()
    g.restore_secondary_values()
    g.update_secondary_values(ddu)
    ff2 = g.assemble_f_int()
    kv2 = g.assemble_kk()
    s2 = g.get_state()
    assert_close(ff1, ff2, tol=1e-13, what="f_int")
    assert_close(kv1, kv2, tol=1e-13, what="K")
    assert_close(s1[0], s2[0], tol=1e-13, what="sigma")
    assert_close(s1[1], s2[1], tol=1e-13, what="[z, lambda]")
    assert np.array_equal(s1[2], s2[2])


@pytest.mark.parametrize("kind", [M.QUA4, M.QUA8, M.HEX8, M.HEX20], ids=["qua4", "qua8", "hex8", "hex20"])
def test_per_cell_calls_match_oracle(kind):
    m, g, o = make(kind, seed=7)
    ddu = plastic_ddu(m, seed=9)
    g.initialize_internal_values()
    g.update_secondary_values(ddu)
    o.initialize()
    o.update_secondary_values(ddu)
    ng, nc = g.ngauss, g.ncomp
    for cell in [0, m.ncell // 2, m.ncell - 1]:
        X = m.coords[m.cells[cell]]
        sl = slice(cell * ng, (cell + 1) * ng)
        kf = oracle.elem_jacobian(kind, ng, X, 1, oracle.Params(E, NU, H, Z0), o.sig[sl], o.ivs[sl], o.elastic[sl])
        assert_close(g.calc_jacobian(cell), kf, what=f"K_e cell {cell}")
        assert_close(g.calc_f_int(cell), oracle.elem_f_int(kind, ng, X, o.sig[sl]), what=f"f_e cell {cell}")


def test_csr_bit_reproducible():
    m, g, o = make(M.HEX20, seed=1)
    ddu = plastic_ddu(m, seed=2)
    g.initialize_internal_values()
    g.backup_secondary_values()
    outs = []
    for _ in range(3):
        ff, kv = np.zeros(g.ndof), np.zeros(g.nnz)
        g.update_and_assemble(ddu, ff, kv)
        outs.append((ff.tobytes(), kv.tobytes()))
    assert outs[0] == outs[1] == outs[2]


@pytest.mark.parametrize("kind", KINDS, ids=[M.KIND_NAMES[k] for k in KINDS])
def test_direct_and_gather_assembly_agree(kind):
    """The direct assembly (blocks added straight into the CSR values and R, every entry summed over
    its cells in the colour-major processing order) gives the same bits on every run, and agrees with
    the gather assembly (upper element-matrix blocks, then row gathers in ascending cell order) to
    1e-13: the summation orders differ and the two are different kernel instantiations, which the
    compiler may contract into fused multiply-adds differently, so only the last bits may differ (a
    missing or doubled block would differ at O(1))."""
    m, g, o = make(kind, seed=7)
    ddu = plastic_ddu(m, seed=8)
    g.initialize_internal_values()
    g.backup_secondary_values()
    got = {}
    for mode in ("direct", "gather", "direct"):
        g.set_assembly(mode)
        ff, kv = np.zeros(g.ndof), np.zeros(g.nnz)
        g.update_and_assemble(ddu, ff, kv)
        f2 = g.assemble_f_int()
        k2 = g.assemble_kk()
        got.setdefault(mode, []).append((ff, kv, f2, k2))
    d0, d1, ga = got["direct"][0], got["direct"][1], got["gather"][0]
    for a, b in zip(d0, d1):
        assert a.tobytes() == b.tobytes(), "direct assembly not reproducible"
    for a, b, what in zip(d0, ga, ("f_int", "K", "f_int (separate)", "K (separate)")):
        assert_close(a, b, tol=1e-13, what=what)
    assert 0 < 1 - g.get_state()[2].mean() < 1


@pytest.mark.parametrize("ngauss", [4, 9])
def test_qua8_gauss_rules(ngauss):
    m, g, o = make(M.QUA8, ngauss=ngauss, seed=4)
    ddu = plastic_ddu(m, seed=4)
    g.initialize_internal_values()
    g.update_secondary_values(ddu)
    o.initialize()
    o.update_secondary_values(ddu)
    sig, ivs, el = g.get_state()
    assert_close(sig, o.sig, what="sigma")
    assert_close(g.assemble_kk(), oracle_csr_values(o, *g.csr_pattern()), what="K")


def test_linear_elastic_and_materials_per_cell():
    """cell_material selects the parameters per cell (cell attribute -> ParamSolid)."""
    from pmsim_b200.elements import Elements, Material
    m = perturbed_mesh(M.QUA8, seed=8, n=(4, 2, 1))
    cm = (np.arange(m.ncell) % 2).astype(np.int32)
    mats = [Material.von_mises(E, NU, H, Z0), Material.linear_elastic(2 * E, 0.25)]
    g = Elements(m, mats, cell_material=cm)
    ddu = plastic_ddu(m, seed=8)
    g.initialize_internal_values()
    g.update_secondary_values(ddu)
    sig, ivs, el = g.get_state()
    ng = g.ngauss
    for c in range(m.ncell):
        model = 1 if cm[c] == 0 else 0
        prm = oracle.Params(E, NU, H, Z0) if model == 1 else oracle.Params(2 * E, 0.25)
        sub = oracle.OracleElements(M.Mesh(2, m.coords, m.cells[c:c + 1], M.QUA8), model, prm)
        sub.initialize()
        sub.update_secondary_values(ddu)
        assert_close(sig[c * ng:(c + 1) * ng], sub.sig, what=f"cell {c}")


def test_errors_are_reported_with_location():
    """A collapsed cell gives the Jacobian error with its cell id (no GPU fault)."""
    from pmsim_b200.elements import Elements, Material
    from pmsim_b200._lib import PmsError
    m = M.structured_2d(M.QUA4, 2, 1, 2.0, 1.0)
    c = m.coords.copy()
    c[m.cells[1][2]] = c[m.cells[1][0]]  # fold cell 1
    g = Elements(M.Mesh(2, c, m.cells, M.QUA4), Material.von_mises(E, NU, H, Z0))
    with pytest.raises(PmsError) as ei:
        g.assemble_kk()
    assert "Jacobian" in str(ei.value)
    assert g.error_location()[0] == 1


def test_femstate_checkpoint_round_trip_on_device():
    """Export the device IP state in pmsim's FemState JSON layout and import it into a fresh handle."""
    from pmsim_b200 import state_io
    m, g, o = make(M.QUA8, seed=12)
    ddu = plastic_ddu(m, seed=12)
    g.initialize_internal_values()
    g.update_secondary_values(ddu)
    text = state_io.export_state(g, u=ddu, ddu=ddu, t=1.0)
    from pmsim_b200.elements import Elements, Material
    h = Elements(m, Material.von_mises(E, NU, H, Z0))
    u, du, t = state_io.import_state(h, text)
    assert t == 1.0 and np.array_equal(u, ddu)
    for a, b in zip(g.get_state(), h.get_state()):
        assert np.array_equal(a, b)
    assert state_io.export_state(h, u=u, ddu=du, t=t) == text


KINDS_2D = [M.TRI3, M.TRI6, M.QUA4, M.QUA8, M.QUA9]


@pytest.mark.parametrize("kind", KINDS_2D, ids=[M.KIND_NAMES[k] for k in KINDS_2D])
def test_axisymmetric_update_and_assemble_matches_oracle(kind):
    """Axisymmetric idealization (x = radius): weight |J| w r, hoop strain u_r/r, hoop rows of B in
    F_int and K (src/base/calculate_strain.rs:36-48, gemlab integrators with args.axisymmetric,
    src/fem/element_solid.rs:128-171), von Mises with plastic and elastic IPs, against the oracle."""
    from pmsim_b200.elements import Elements, Material
    m = perturbed_mesh(kind, seed=7, n=GRID[2])
    m.coords[:, 0] += 0.5  # keep every point off the axis
    g = Elements(m, Material.von_mises(E, NU, H, Z0), axisymmetric=True)
    o = oracle.OracleElements(m, 1, oracle.Params(E, NU, H, Z0), sym_tol=-1.0, axisymmetric=True)
    indptr, indices = g.csr_pattern()
    g.initialize_internal_values()
    o.initialize()
    assert_close(g.assemble_kk(), oracle_csr_values(o, indptr, indices), what="K elastic")
    ddu = plastic_ddu(m, seed=kind + 40)
    g.backup_secondary_values()
    ff = np.zeros(g.ndof)
    kv = np.zeros(g.nnz)
    g.update_and_assemble(ddu, ff, kv)
    o.update_secondary_values(ddu)
    sig, ivs, el = g.get_state()
    assert np.array_equal(el, o.elastic), "elastic flags differ"
    assert 0 < (1 - el.mean()) < 1, "expected a mix of elastic and plastic IPs"
    assert_close(sig, o.sig, what="sigma")
    assert_close(ivs, o.ivs, what="[z, lambda]")
    assert_close(ff, o.assemble_f_int(), what="f_int")
    assert_close(kv, oracle_csr_values(o, indptr, indices), what="K")


def test_sgm_5d17_axisymmetric_on_device():
    """tests/test_solid_smith_5d17_qua4_axisym.rs on the device elements (two layers, 9 IP, point
    loads, reduced-system method): the reference test's displacements at its tolerance 1e-9."""
    import problems
    from pmsim_b200.elements import Elements, Material
    from pmsim_b200.solver import SolverImplicit
    pb = problems.sgm_5d17_axisym()
    mats = [Material.linear_elastic(E_, nu) for E_, nu in pb["mats"]]
    el = Elements(pb["mesh"], mats, ngauss=9, cell_material=pb["cmat"], axisymmetric=True)
    sol = SolverImplicit(el, pb["essential"], loads=pb["loads"], lagrange_mult_method=False, t_fin=1.0)
    out = {}
    sol.solve(lambda step, t, u, e: out.setdefault("u", u.copy()))
    np.testing.assert_allclose(out["u"], pb["golden"]["uu_correct"], rtol=0, atol=1e-9)


@pytest.mark.parametrize("kind", KINDS_2D, ids=[M.KIND_NAMES[k] for k in KINDS_2D])
def test_plane_stress_update_and_assemble_matches_oracle(kind):
    """Plane stress (linear elastic; in-plane normal block E/(1-nu^2) (1, nu; nu, 1), no sigma_zz) with
    thickness 0.25, against the oracle."""
    from pmsim_b200.elements import Elements, Material
    m = perturbed_mesh(kind, seed=9, n=GRID[2])
    g = Elements(m, Material.linear_elastic(E, NU), thickness=0.25, plane_stress=True)
    o = oracle.OracleElements(m, oracle.MODEL_LINEAR_ELASTIC_PLANE_STRESS, oracle.Params(E, NU, 0.0, 1.0), thickness=0.25)
    indptr, indices = g.csr_pattern()
    g.initialize_internal_values()
    o.initialize()
    ddu = plastic_ddu(m, seed=kind + 60)
    g.backup_secondary_values()
    ff = np.zeros(g.ndof)
    kv = np.zeros(g.nnz)
    g.update_and_assemble(ddu, ff, kv)
    o.update_secondary_values(ddu)
    sig = g.get_state()[0]
    assert np.all(sig[:, 2] == 0.0), "plane stress keeps sigma_zz = 0"
    assert_close(sig, o.sig, what="sigma")
    assert_close(ff, o.assemble_f_int(), what="f_int")
    assert_close(kv, oracle_csr_values(o, indptr, indices), what="K")


def test_bhatti_1d6_plane_stress_on_device():
    """tests/test_solid_bhatti_1d6_plane_stress.rs on the device elements: the reference test's
    displacements (its tolerance is 1e-15; the device sums in another order, so 1e-14 here)."""
    import problems
    from pmsim_b200.elements import Elements, Material
    from pmsim_b200.solver import SolverImplicit
    pb = problems.bhatti_1d6_plane_stress()
    el = Elements(pb["mesh"], Material.linear_elastic(pb["young"], pb["poisson"]), thickness=pb["thickness"],
                  plane_stress=True)
    sol = SolverImplicit(el, pb["essential"], lagrange_mult_method=False, t_fin=1.0, natural=pb["natural"])
    out = {}
    sol.solve(lambda step, t, u, e: out.setdefault("u", u.copy()))
    np.testing.assert_allclose(out["u"], pb["golden"]["uu_correct"], rtol=0, atol=1e-14)


@pytest.mark.parametrize("kind,ngauss,n", [(M.HEX8, 8, (1, 1, 1)), (M.HEX8, 8, (2, 1, 1)), (M.HEX8, 8, (7, 1, 1)),
                                           (M.HEX8, 1, (5, 2, 1)), (M.HEX8, 27, (5, 2, 1)), (M.HEX8, 8, (18, 18, 17)),
                                           (M.TET4, 1, (1, 1, 1)), (M.TET4, 4, (1, 1, 1)), (M.TET4, 4, (3, 1, 3)),
                                           (M.TET4, 4, (13, 12, 16))])
def test_cells_packed_into_warps(kind, ngauss, n):
    """Hex8 and Tet4 run three and eight cells to a warp: one cell, ragged last groups, more groups than
    the device holds at once, and the rules that fit the slots and that do not, against the oracle at the
    parity tolerance (the separate calls too)."""
    from pmsim_b200.elements import Elements, Material
    m = perturbed_mesh(kind, seed=3, n=n)
    g = Elements(m, Material.von_mises(E, NU, H, Z0), ngauss=ngauss)
    o = oracle.OracleElements(m, 1, oracle.Params(E, NU, H, Z0), ngauss=ngauss, sym_tol=-1.0, nthreads=0)
    indptr, indices = g.csr_pattern()
    ddu = plastic_ddu(m, seed=4)
    g.initialize_internal_values()
    o.initialize()
    g.backup_secondary_values()
    ff, kv = np.zeros(g.ndof), np.zeros(g.nnz)
    g.update_and_assemble(ddu, ff, kv)
    o.update_secondary_values(ddu)
    sig, ivs, el = g.get_state()
    assert np.array_equal(el, o.elastic)
    assert_close(sig, o.sig, what="sigma")
    assert_close(ivs, o.ivs, what="[z, lambda]")
    fo, ko = o.assemble_f_int(), oracle_csr_values(o, indptr, indices)
    assert_close(ff, fo, what="f_int")
    assert_close(kv, ko, what="K")
    assert_close(g.assemble_f_int(), fo, what="f_int alone")
    assert_close(g.assemble_kk(), ko, what="K alone")


@pytest.mark.parametrize("kind", [M.QUA8, M.TRI3, M.HEX8], ids=["qua8", "tri3", "hex8"])
def test_values_that_start_on_an_odd_eight_bytes(kind):
    """The CSR values may start anywhere a double may: the same bits as at a 16-byte boundary."""
    import torch
    m, g, _ = make(kind, seed=6)
    g.initialize_internal_values()
    g.backup_secondary_values()
    ddu = torch.tensor(plastic_ddu(m, seed=7), device="cuda")
    out = []
    for shift in (0, 1):
        ff = torch.zeros(g.ndof, dtype=torch.float64, device="cuda")
        kv = torch.zeros(g.nnz + 2, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        g.update_and_assemble(ddu, ff, kv[shift:shift + g.nnz])
        g.sync()
        out.append((ff.cpu().numpy(), kv[shift:shift + g.nnz].cpu().numpy()))
        assert float(kv[:shift].abs().sum()) == 0.0 and float(kv[shift + g.nnz:].abs().sum()) == 0.0
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])


@pytest.mark.parametrize("kind,n", [(M.QUA8, (20, 21, 1)), (M.QUA8, (60, 40, 1)), (M.HEX20, (7, 6, 5))],
                         ids=["below one piece", "about one piece", "several pieces"])
def test_host_arrays_pageable_pinned_and_device(kind, n):
    """K into pageable memory (in pinned pieces of 262,144 values once it is that large), into pinned
    memory and on the device: the same bits, for both triangles' storage and one's."""
    import torch
    m = perturbed_mesh(kind, seed=2, n=n)
    from pmsim_b200.elements import Elements, Material
    g = Elements(m, Material.von_mises(E, NU, H, Z0))
    g.initialize_internal_values()
    g.backup_secondary_values()
    ddu = plastic_ddu(m, seed=3)
    for sym in ("full", "lower"):
        g.set_symmetry(sym)
        d_kv = torch.zeros(g.nnz, dtype=torch.float64, device="cuda")
        d_ff = torch.zeros(g.ndof, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        g.update_and_assemble(torch.tensor(ddu, device="cuda"), d_ff, d_kv)
        g.sync()
        for kv in (np.zeros(g.nnz), torch.zeros(g.nnz, dtype=torch.float64).pin_memory().numpy()):
            ff = np.zeros(g.ndof)
            g.update_and_assemble(ddu, ff, kv)
            assert np.array_equal(kv, d_kv.cpu().numpy()) and np.array_equal(ff, d_ff.cpu().numpy())


@pytest.mark.parametrize("kind,ngauss,n", [(M.TET4, 4, (2, 2, 2)), (M.TET4, 4, (7, 6, 5)), (M.HEX8, 8, (2, 2, 2)),
                                           (M.HEX8, 8, (9, 8, 7)), (M.HEX8, 8, (19, 18, 18)),
                                           (M.HEX20, 8, (3, 2, 2)), (M.HEX20, 8, (6, 6, 6))])
@pytest.mark.parametrize("sym", ["full", "lower"])
def test_gather_of_few_rows(kind, ngauss, n, sym):
    """The gather loads further ahead where all rows are in flight at once: rows of one cell and of many,
    numbers of cells that are no multiple of the cells loaded together, and a mesh past the line, against
    the oracle at the parity tolerance."""
    from pmsim_b200.elements import Elements, Material
    m = perturbed_mesh(kind, seed=5, n=n)
    g = Elements(m, Material.von_mises(E, NU, H, Z0), ngauss=ngauss)
    o = oracle.OracleElements(m, 1, oracle.Params(E, NU, H, Z0), ngauss=ngauss, sym_tol=-1.0, nthreads=0)
    indptr, indices = g.csr_pattern()
    ddu = plastic_ddu(m, seed=6)
    g.initialize_internal_values()
    o.initialize()
    g.backup_secondary_values()
    g.set_symmetry(sym)
    ff, kv = np.zeros(g.ndof), np.zeros(g.nnz)
    g.update_and_assemble(ddu, ff, kv)
    o.update_secondary_values(ddu)
    ko = oracle_csr_values(o, indptr, indices)
    if sym == "lower":
        rows = np.repeat(np.arange(len(indptr) - 1), np.diff(indptr))
        ko = ko[np.asarray(indices) <= rows]
    assert_close(ff, o.assemble_f_int(), what="f_int")
    assert_close(kv, ko, what="K")


@pytest.mark.parametrize("kind,ngauss,n", [(M.QUA8, 9, (20, 10, 1)), (M.TRI6, 3, (9, 8, 1)), (M.TET4, 4, (4, 3, 3)),
                                           (M.HEX8, 8, (6, 5, 5)), (M.HEX20, 27, (3, 3, 2)),
                                           (M.QUA8, 9, (60, 45, 1)), (M.TET4, 4, (13, 13, 12)), (M.HEX8, 8, (11, 10, 10))],
                         ids=["qua8", "tri6", "tet4", "hex8", "hex20", "qua8 more blocks than SMs", "tet4 more", "hex8 more"])
def test_calls_that_follow_one_another_without_a_wait(kind, ngauss, n):
    """On small meshes the kernels of successive calls overlap their launches while the element matrices are
    written again and again: K and R of many calls in a row, each with another increment (and F_int alone
    in between), are the bits of the same calls made one at a time."""
    import torch
    from pmsim_b200.elements import Elements, Material
    m = perturbed_mesh(kind, seed=8, n=n)
    g = Elements(m, Material.von_mises(E, NU, H, Z0), ngauss=ngauss)
    g.initialize_internal_values()
    g.backup_secondary_values()
    count = 60
    ddu = [torch.tensor(plastic_ddu(m, seed=10 + k) * (0.2 + 0.05 * k), device="cuda") for k in range(count)]
    runs = []
    for wait in (True, False):
        ff = torch.zeros(count, g.ndof, dtype=torch.float64, device="cuda")
        f2 = torch.zeros(count, g.ndof, dtype=torch.float64, device="cuda")
        kk = torch.zeros(count, g.nnz, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        for k in range(count):
            g.update_and_assemble(ddu[k], ff[k], kk[k])
            if wait:
                g.sync()
            if k % 3 == 2:
                g.assemble_f_int(f2[k])
                if wait:
                    g.sync()
        g.sync()
        runs.append((ff.cpu().numpy(), f2.cpu().numpy(), kk.cpu().numpy()))
    for a, b in zip(*runs):
        assert np.array_equal(a, b)
    assert not np.array_equal(runs[0][2][0], runs[0][2][-1])  # (the first increments are elastic)


def test_state_is_read_while_another_device_is_current():
    """get_state needs no particular current device, leaves the one it finds current, and gives what it gives
    on the handle's own."""
    import torch
    if torch.cuda.device_count() < 2:
        pytest.skip("one GPU")
    m, g, _ = make(M.HEX8, seed=9)
    g.initialize_internal_values()
    g.update_secondary_values(plastic_ddu(m, seed=10))
    g.sync()
    with torch.cuda.device(1):
        first = g.get_state()  # (its scratch is made here)
        again = g.get_state()
        assert torch.cuda.current_device() == 1
        torch.zeros(1, device="cuda").add_(1.0)
    for a, b, c in zip(first, again, g.get_state()):
        assert np.array_equal(a, b) and np.array_equal(a, c)


@pytest.mark.parametrize("want", [(1, 1, 1), (1, 0, 0), (0, 1, 0), (0, 0, 1), (0, 0, 0)])
def test_state_arrays_are_optional(want):
    """Any of the three arrays of pms_elements_get_state may be null; the others are the same."""
    from pmsim_b200 import _lib
    m, g, _ = make(M.QUA8, seed=9)
    g.initialize_internal_values()
    g.update_secondary_values(plastic_ddu(m, seed=10))
    full = g.get_state()
    arrays = [np.full_like(a, 7) for a in full]
    rc = g.L.pms_elements_get_state(g.h, *(_lib.ptr(a) if w else None for a, w in zip(arrays, want)))
    assert rc == 0
    for a, f, w in zip(arrays, full, want):
        assert np.array_equal(a, f if w else np.full_like(f, 7))
