"""cfd_rhs_noalloc without wiring tables (every type a configuration can wire
by itself, and DoubleMachUp, which keeps the table) against cfd_rhs of a handle
with the same configuration: the same kernels on the same ghosts, so the
right-hand sides agree bit for bit."""
import ctypes as C

import numpy as np
import pytest

from cfd_inwsl_b200 import _lib, zone
from tests.util import make_info

pytestmark = pytest.mark.gpu
B = zone.BndType


@pytest.mark.parametrize("n,bc", [
    ((131,), [[B.SUPERSONICOUTLET, B.SYMMETRY1D]]),
    ((131,), [[B.PERIODIC_WRAP] * 2]),
    ((37, 21), [[B.PERIODIC1D, B.SYMMETRYX], [B.SYMMETRYY, B.SUPERSONICOUTLET]]),
    ((37, 21), [[B.PERIODIC_WRAP] * 2, [B.PERIODIC_WRAP] * 2]),
    ((40, 24), [[B.SUPERSONICOUTLET] * 2, [B.SYMMETRYY, B.DoubleMachUp]]),
    ((9, 17, 11), [[B.SYMMETRYX, B.PERIODIC1D], [B.SYMMETRYY] * 2, [B.SYMMETRYZ, B.SUPERSONICOUTLET]]),
    ((9, 17, 11), [[B.PERIODIC_WRAP] * 2] * 3)])
@pytest.mark.parametrize("strict", [True, False])
def test_noalloc_matches_handle(n, bc, strict):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    rng = np.random.default_rng(sum(n))
    dim, nc = len(n), int(np.prod(n))
    prim = np.concatenate([rng.uniform(0.5, 2, (1, nc)), rng.uniform(-1, 1, (dim, nc)), rng.uniform(0.5, 2, (1, nc))])
    info = make_info(dim, list(n), [0, 1, 0, 1, 0, 1], 2, 0, strict)
    bc3 = bc + [[B.SUPERSONICOUTLET] * 2] * (3 - dim)
    s = zone.BlockSolver(info, bc=bc3)
    s.set_cons(zone.prim_to_cons(prim.T))
    info.t = 0.03
    want = s.rhsSolve()
    u = torch.from_numpy(np.ascontiguousarray(s.cons.T)).cuda()
    out = torch.empty_like(u)
    st = torch.cuda.current_stream().cuda_stream
    _lib.check(s.lib.cfd_rhs_noalloc(C.byref(s.cfg), C.c_void_p(u.data_ptr()), C.c_void_p(out.data_ptr()), 0.03,
                                     C.c_void_p(st)))
    torch.cuda.synchronize()
    s.close()
    np.testing.assert_array_equal(out.cpu().numpy().T, want)
