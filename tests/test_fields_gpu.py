"""Fields across the API: values in and out of every solver's device layout in
pieces, whatever the field's size, and with a bounded amount of device memory
beside the fields themselves."""
import os

import numpy as np
import pytest

import emsolvers_gb300 as ems

pytestmark = pytest.mark.gpu
EPS0, MU0 = 8.8541878128e-12, 1.25663706212e-6
H = 1e-3
DT = 0.05 * H / 299792458.0
KDIR = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "kmat")
# the largest scratch buffer of a handle's field copies (2^20 values), and what
# the allocator rounds up to
SCRATCH = (1 << 20) * 8 + (4 << 20)


def _handle(kind, prec):
    if kind == "fdtd":
        return ems.FdtdSimulation((200, 180, 170), H, DT, EPS0, MU0, 1, prec), 6
    if kind == "hex":
        return ems.HexFemSimulation(1, (121, 110, 105), H, DT, EPS0, MU0, 1, True, ems.SYMP2, prec, KDIR), 3
    if kind == "tet1":
        return ems.TetFemSimulation((90, 85, 80), H, 1, ems.SYMP2, prec, dt=DT), 2
    return ems.TetFemBatch([(40, 41, 42), (30, 50, 40)], H, order=2, integrator=ems.SYMP2, precision=prec, dt=DT), 2


@pytest.mark.parametrize("prec", [ems.FP64, ems.FP32], ids=["fp64", "fp32"])
@pytest.mark.parametrize("kind", ["fdtd", "hex", "tet1", "tet2"])
def test_fields_of_several_pieces_in_bounded_memory(kind, prec):
    torch = pytest.importorskip("torch")
    s, nf = _handle(kind, prec)
    rng = np.random.default_rng(3)
    sizes = [s.field_size(q) for q in range(nf)]
    assert max(sizes) > (1 << 21)   # more than two pieces
    # values exact in FP32, which every field keeps (order-2 tetrahedra hold their dead DOFs at zero)
    vals = [rng.standard_normal(n).astype(np.float32).astype(np.float64) for n in sizes]
    free = torch.cuda.mem_get_info()[0]
    for q in range(nf):
        s.set_field(q, vals[q])
    for q in range(nf):
        got = s.get_field(q)
        live = got != 0 if kind == "tet2" else np.ones(sizes[q], bool)
        assert live.mean() > 0.8
        assert np.array_equal(got[live], vals[q][live])
    assert free - torch.cuda.mem_get_info()[0] <= SCRATCH
    s.close()


@pytest.mark.parametrize("prec", [ems.FP64, ems.FP32], ids=["fp64", "fp32"])
@pytest.mark.parametrize("kind", ["fdtd", "hex", "tet1", "tet2"])
def test_threads_read_fields_of_one_handle(kind, prec):
    """Threads that read fields of the same handle at the same time each get
    their own field."""
    from concurrent.futures import ThreadPoolExecutor
    s, nf = _handle(kind, prec)
    rng = np.random.default_rng(4)
    for q in range(nf):
        s.set_field(q, rng.standard_normal(s.field_size(q)))
    ref = [s.get_field(q) for q in range(nf)]
    with ThreadPoolExecutor(4) as ex:
        for q, got in zip(list(range(nf)) * 6, ex.map(s.get_field, list(range(nf)) * 6)):
            assert np.array_equal(got, ref[q])
    s.close()
