"""Device-resident traces: a WEMVA call carries no `data`, only `wemvaData`."""
import ctypes as C

import numpy as np
import pytest

from cases import make_case

pytestmark = pytest.mark.gpu


def test_wemva_adjoint_without_data_traces():
    """The plan timing of a WEMVA call injects its own traces: `data` is NULL in device memory. The
    grid is this test's own, so that no plan measured by another context is reused."""
    import torch

    import orc
    from acoustic_isotropic_operators_b200.batch import Context, Shot
    c = make_case(seed=4, nzi=52, nxi=68, nts=40, sub=4, nExt=5, nshots=2)
    s = c.scheme
    k = orc.constants(s, c.vel, dtype=np.float32)
    data = [(c.rng.standard_normal((len(r), s.nts)) * 1e-2).astype(np.float32) for r in c.rec_pos]
    ext = np.zeros((5, s.nx, s.nz), np.float32)
    ext[:, 5:-5, 5:-5] = c.rng.standard_normal((5, s.nx - 10, s.nz - 10))
    ctx = Context(s.nz, s.nx, s.nts, s.dts, s.sub, s.dz, s.dx, s.minPad, k["v2"], k["rs"], nExt=5)
    dev = [(torch.from_numpy(c.sig[i]).cuda(), torch.from_numpy(data[i]).cuda()) for i in range(2)]
    e, out = torch.from_numpy(ext).cuda(), torch.zeros((s.nx, s.nz), device="cuda")
    torch.cuda.synchronize()
    ctx.device_call("wemva_ext_adjoint", C.c_void_p(out.data_ptr()), C.c_int(0), C.c_void_p(e.data_ptr()),
                    shots=[(c.src_pos[i], c.rec_pos[i], dev[i][0].data_ptr(), 0, dev[i][1].data_ptr(), 0) for i in range(2)])
    host = ctx.wemva_adjoint(ext, [Shot(c.src_pos[i], c.rec_pos[i], c.sig[i], None, data[i]) for i in range(2)])
    ctx.close()
    assert np.abs(host).max() > 0
    np.testing.assert_array_equal(out.cpu().numpy(), host)
