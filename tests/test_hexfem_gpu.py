"""Hexahedral FEM (fem_v2 leapfrog, symplectic_2, symplectic_4; orders 1-3)
on the GPU through the C ABI.  FP64 must equal the reference bit for bit
(golden fixtures); FP32 is compared with the FP64 reference by relative L2
error, tolerance 1e-4 on traces and fields."""
import numpy as np
import pytest

import golden_io
import oracle
from gpu_util import rel_l2
import emsolvers_gb300 as ems

pytestmark = pytest.mark.gpu
INTEG = {"fem_v2": ems.LEAPFROG, "symplectic_2": ems.SYMP2, "symplectic_4": ems.SYMP4}
FP32_TOL = 1e-4


def _run(m, precision):
    s = ems.HexFemSimulation(m["order"], m["grid"], m["h"], m["dt"], m["eps"], m["mu"], m["tf"], m["use_ofem"],
                             integrator=INTEG[m["variant"]], precision=precision, kmat_dir=golden_io.KMAT_DIR)
    [s.setSource_x, s.setSource_y, s.setSource_z][m["source"][0]](m["source"][1])
    s.setObservationPoint(m["observation"])
    s.run(m["nsteps"])
    return s.traces()[0], s.levels()


@pytest.mark.parametrize("case", list(golden_io.femv2_cases()), ids=lambda c: c[0]["name"])
def test_fp64_bitwise_equal_to_reference(case):
    m, tr, ef = case
    t, lv = _run(m, ems.FP64)
    np.testing.assert_array_equal(t, tr)
    for q in range(3):
        np.testing.assert_array_equal(lv[q], ef[q])


@pytest.mark.parametrize("case", list(golden_io.femv2_cases()), ids=lambda c: c[0]["name"])
def test_fp32_within_tolerance_of_reference(case):
    m, tr, ef = case
    t, lv = _run(m, ems.FP32)
    assert rel_l2(t[:, 1:], tr[:, 1:]) < FP32_TOL
    assert np.array_equal(t[:, 0], tr[:, 0])
    # compare all stored levels, normalised by the norm of all components
    num = sum(np.sum((lv[q] - ef[q]) ** 2) for q in range(3))
    den = sum(np.sum(ef[q] ** 2) for q in range(3))
    assert np.sqrt(num / den) < FP32_TOL


@pytest.mark.parametrize("order", [1, 2])
@pytest.mark.parametrize("integ", [oracle.SYMP2, oracle.SYMP4, oracle.LEAPFROG])
def test_fp64_longer_run_matches_oracle(order, integ):
    g = (8 * order, 6 * order, 6 * order) if order == 1 else (8, 8, 10)
    h = 0.05
    c0 = 1 / np.sqrt(8.8541878128e-12 * 1.25663706212e-6)
    dt = h / (c0 * np.sqrt(3.0)) / 2.0
    km = oracle.load_kmat(golden_io.kmat_path(order, 1))
    src = (2, (g[0] // 2, g[1] // 2, g[2] // 2))
    obs = [(g[0] // 2 + 1, g[1] // 2, g[2] // 2), (2, 2, 2)]
    tr_o, ef_o = oracle.hexfem_run(order, g, h, dt, 8.8541878128e-12, 1.25663706212e-6, 3, integ, km, 120, [src], obs)
    s = ems.HexFemSimulation(order, g, h, dt, 8.8541878128e-12, 1.25663706212e-6, 3, 1, integrator=integ,
                             precision=ems.FP64, kmat_dir=golden_io.KMAT_DIR)
    s.setSource_z(src[1])
    for o in obs:
        s.setObservationPoint(o)
    s.run(120)
    np.testing.assert_array_equal(s.traces(), tr_o)
    for q, lv in enumerate(s.levels()):
        np.testing.assert_array_equal(lv, ef_o[q])


def test_save_results_format(tmp_path):
    m, tr, _ = next(iter(golden_io.femv2_cases()))
    s = ems.HexFemSimulation(m["order"], m["grid"], m["h"], m["dt"], m["eps"], m["mu"], m["tf"], m["use_ofem"],
                             kmat_dir=golden_io.KMAT_DIR)
    s.setSource_z(m["source"][1])
    s.setObservationPoint(m["observation"])
    s.run(m["nsteps"])
    fn = tmp_path / "out.csv"
    s.saveResults(m["nsteps"], str(fn))
    lines = fn.read_text().splitlines()
    assert lines[0] == "time,Ex,Ey,Ez"
    vals = np.array([[float(v) for v in l.split(",")] for l in lines[1:]])
    np.testing.assert_allclose(vals, tr, rtol=1e-14, atol=0)
    assert "e" in lines[2]  # scientific, 15 digits


@pytest.mark.parametrize("ofem", [1, 0])
@pytest.mark.parametrize("order,grid", [(1, (2, 2, 2)), (1, (5, 3, 4)), (1, (33, 2, 7)), (1, (17, 15, 17)), (2, (4, 4, 4)), (2, (5, 7, 6)), (2, (34, 4, 6)),
                                        (2, (9, 8, 11))])
@pytest.mark.parametrize("integ", [oracle.LEAPFROG, oracle.SYMP4])
def test_two_pass_force_bitwise_equal_to_oracle(order, grid, integ, ofem):
    """Element pass and DOF pass against the oracle's element loop: grids of
    two elements a side and odd ones, grid lines beyond the last whole element
    (order 2 on odd grids), sources on inner, outer and shared edges, sampling
    every second step over replayed and single steps, continued in a second
    run."""
    if order == 2 and not ofem:
        pytest.skip("no lumped order-2 matrix among the fixtures")
    h, eps, mu = 0.05, 8.8541878128e-12, 1.25663706212e-6
    dt = h * np.sqrt(eps * mu / 3.0) / 2.0
    km = oracle.load_kmat(golden_io.kmat_path(order, ofem))
    srcs = [(2, (grid[0] // 2, grid[1] // 2, grid[2] // 2)), (0, (0, 1, 1)), (1, (1, 0, grid[2] - 1))]
    obs = [(grid[0] // 2, grid[1] // 2, grid[2] // 2), (1, 1, 0)]
    steps = 23
    tr_o, ef_o = oracle.hexfem_run(order, grid, h, dt, eps, mu, 2, integ, km, steps, srcs, obs)
    s = ems.HexFemSimulation(order, grid, h, dt, eps, mu, 2, ofem, integrator=integ, precision=ems.FP64, kmat_dir=golden_io.KMAT_DIR)
    for c, at in srcs:
        (s.setSource_x, s.setSource_y, s.setSource_z)[c](at)
    for o in obs:
        s.setObservationPoint(o)
    s.run(steps)
    np.testing.assert_array_equal(s.traces(), tr_o)
    for q, lv in enumerate(s.levels()):
        np.testing.assert_array_equal(lv, ef_o[q])
    t1, l1 = s.traces(), s.levels()
    s.reset()
    s.run(10)
    s.run(steps - 10)
    np.testing.assert_array_equal(s.traces()[:, :, 1:], t1[:, 5:, 1:])
    for q, lv in enumerate(s.levels()):
        np.testing.assert_array_equal(lv, l1[q])


def test_grid_beyond_32_bit_dof_indices():
    """A component of more than 2^31 DOFs (a rod of 2 x 2 x 240 million
    elements): a wave launched just below DOF 2^31 and crossing it gives the
    bits of the same wave in a short rod whose ends it does not reach."""
    torch = pytest.importorskip("torch")
    if torch.cuda.mem_get_info()[0] < 100e9:
        pytest.skip("needs 100 GB of device memory")
    h, eps, mu = 0.05, 8.8541878128e-12, 1.25663706212e-6
    dt = h * np.sqrt(eps * mu / 3.0) / 2.0
    nz, steps = 240_000_000, 24
    top = (2 ** 31 - 1) // 9 - 2            # Ez has 3 x 3 values per layer
    assert 9 * nz > 2 ** 31 and 9 * (top + 1) < 2 ** 31 < 9 * (top + 12)

    def run(grid, z):
        s = ems.HexFemSimulation(1, grid, h, dt, eps, mu, 1, 1, precision=ems.FP32, kmat_dir=golden_io.KMAT_DIR)
        s.setSource_z((1, 1, z))
        for q in (z - 5, z - 1, z):
            s.setObservationPoint((1, 1, q))
        s.run(steps)
        t = s.traces()
        s.close()
        return t

    ref, got = run((2, 2, 400), 200), run((2, 2, nz), top)
    assert np.abs(ref[..., 1:]).max() > 0
    np.testing.assert_array_equal(got, ref)


@pytest.mark.parametrize("grid", [(28, 28, 29), (31, 29, 30), (61, 20, 20)])
@pytest.mark.parametrize("integ", [oracle.LEAPFROG, oracle.SYMP4])
def test_order2_fp64_on_both_sides_of_the_one_pass_rule_bitwise_equal_to_oracle(grid, integ):
    """FP64 of order 2 sums DOF by DOF on grids of fewer than 3000 elements
    (2744 here) and in two passes on larger ones (3150 and 3000, odd grid lines
    among them): the oracle's bits from either."""
    h, eps, mu = 0.05, 8.8541878128e-12, 1.25663706212e-6
    dt = h * np.sqrt(eps * mu / 3.0) / 2.0
    km = oracle.load_kmat(golden_io.kmat_path(2, 1))
    srcs = [(2, tuple(v // 2 for v in grid)), (0, (0, 1, 1))]
    obs = [tuple(v // 2 for v in grid)]
    steps = 12
    tr_o, ef_o = oracle.hexfem_run(2, grid, h, dt, eps, mu, 2, integ, km, steps, srcs, obs)
    s = ems.HexFemSimulation(2, grid, h, dt, eps, mu, 2, 1, integrator=integ, precision=ems.FP64, kmat_dir=golden_io.KMAT_DIR)
    for c, at in srcs:
        (s.setSource_x, s.setSource_y, s.setSource_z)[c](at)
    s.setObservationPoint(obs[0])
    s.run(steps)
    np.testing.assert_array_equal(s.traces(), tr_o)
    for q, lv in enumerate(s.levels()):
        np.testing.assert_array_equal(lv, ef_o[q])
    name = s.time_dominant_kernel(1)[2]
    assert ("elem" in name) == (np.prod([v // 2 for v in grid]) >= 3000), name


@pytest.mark.parametrize("integ", [ems.LEAPFROG, ems.SYMP4])
def test_no_room_for_the_element_values(integ):
    """A grid whose fields fit while the two passes' element values do not
    (384 MB here, 150 MB left): the run takes the one-pass kernels and gives the
    same bits."""
    torch = pytest.importorskip("torch")
    g, h, eps, mu = (200, 200, 200), 0.05, 8.8541878128e-12, 1.25663706212e-6
    dt = h * np.sqrt(eps * mu / 3.0) / 2.0
    out = []
    for full in (False, True):
        s = ems.HexFemSimulation(1, g, h, dt, eps, mu, 1, 1, integrator=integ, precision=ems.FP32, kmat_dir=golden_io.KMAT_DIR)
        s.setSource_z((100, 100, 100))
        s.setObservationPoint((101, 100, 100))
        hog = torch.empty(torch.cuda.mem_get_info()[0] - (150 << 20), dtype=torch.uint8, device="cuda") if full else None
        s.run(11)
        out.append((s.traces(), s.get_field(2)))
        del hog
        torch.cuda.empty_cache()
        s.close()
    assert np.linalg.norm(out[0][1]) > 0
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("integ", [ems.LEAPFROG, ems.SYMP2, ems.SYMP4])
@pytest.mark.parametrize("order,prec", [(1, ems.FP64), (1, ems.FP32), (2, ems.FP32)])
def test_replayed_steps_over_runs_equal_single_steps(order, prec, integ):
    """Runs that begin at every position of the leapfrog ring, repeated runs that
    replay a kept graph, and sources and receivers added between runs: the bits
    of the same steps run one by one."""
    g, h, eps, mu = (12, 9, 10), 0.05, 8.8541878128e-12, 1.25663706212e-6
    dt = h * np.sqrt(eps * mu / 3.0) / 2.0
    out = []
    for single in (False, True):
        s = ems.HexFemSimulation(order, g, h, dt, eps, mu, 1, 1, integrator=integ, precision=prec, kmat_dir=golden_io.KMAT_DIR)

        def run(n):
            t = []
            for k in [1] * n if single else [n]:
                s.run(k)
                t.append(s.traces())
            return np.concatenate(t, axis=1)

        tr = []
        s.setSource_z((6, 4, 5))
        s.setObservationPoint((5, 4, 4))
        tr += [run(17), run(17), run(17), run(100)]
        s.setSource_x((3, 4, 5))
        tr += [run(100), run(100)]
        s.setObservationPoint((7, 3, 5))
        tr += [run(100), run(17)]
        out.append((tr, s.levels()))
        s.close()
    assert np.abs(out[0][0][-1][..., 1:]).max() > 0
    for a, b in zip(out[0][0], out[1][0]):
        np.testing.assert_array_equal(a, b)
    for a, b in zip(out[0][1], out[1][1]):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("ofem", [1, 0])
@pytest.mark.parametrize("grid", [(21, 21, 22), (33, 31, 10), (25, 20, 20)])
@pytest.mark.parametrize("integ", [oracle.LEAPFROG, oracle.SYMP2])
def test_order1_fp64_element_passes_bitwise_equal_to_oracle(grid, integ, ofem):
    """Grids of 9702, 10230 and 10000 elements, on both sides of the line from
    which one thread takes a whole element of order 1 in FP64."""
    h, eps, mu = 0.05, 8.8541878128e-12, 1.25663706212e-6
    dt = h * np.sqrt(eps * mu / 3.0) / 2.0
    km = oracle.load_kmat(golden_io.kmat_path(1, ofem))
    srcs = [(2, tuple(v // 2 for v in grid)), (0, (0, 1, 1))]
    obs = [tuple(v // 2 for v in grid), (1, 1, 0)]
    tr_o, ef_o = oracle.hexfem_run(1, grid, h, dt, eps, mu, 2, integ, km, 25, srcs, obs)
    s = ems.HexFemSimulation(1, grid, h, dt, eps, mu, 2, ofem, integrator=integ, precision=ems.FP64, kmat_dir=golden_io.KMAT_DIR)
    for c, at in srcs:
        (s.setSource_x, s.setSource_y, s.setSource_z)[c](at)
    for o in obs:
        s.setObservationPoint(o)
    s.run(25)
    np.testing.assert_array_equal(s.traces(), tr_o)
    for q, lv in enumerate(s.levels()):
        np.testing.assert_array_equal(lv, ef_o[q])
