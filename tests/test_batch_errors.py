"""A batch call that the runtime refuses reports it once: the next call of the thread succeeds."""
from __future__ import annotations

import ctypes as C

import pytest

pytestmark = pytest.mark.gpu


def test_error_does_not_outlive_the_call(f3d, cuda_ok):
    import torch
    rt = pytest.importorskip("cuda.bindings.runtime")
    S, B = f3d.solver_module(), f3d.batch_module()
    dcs = [S.DeviceCase(f3d.random_curvilinear(n=8, ns=ns, seed=ns), tile=3) for ns in (1, 2)]
    b = B.Batch(dcs, mode="persistent")  # two species counts: two lanes
    lib = f3d.load_library()
    torch.cuda.synchronize()
    st = torch.cuda.Stream()
    # a capture that a synchronisation has invalidated refuses every further call on its stream
    rt.cudaStreamBeginCapture(st.cuda_stream, rt.cudaStreamCaptureMode.cudaStreamCaptureModeRelaxed)
    rt.cudaStreamSynchronize(st.cuda_stream)
    rc = lib.flame_batch_stage(b.handle, C.c_void_p(st.cuda_stream), 1, 0)
    msg = f3d.abi.last_error(lib)
    rt.cudaStreamEndCapture(st.cuda_stream)
    assert rc == 2 and "flame_batch_stage" in msg
    dcs[0]._call("flame_prim2c", dcs[0].U.data_ptr(), dcs[0].Q[0].data_ptr())
    b.step()
    b.status()
    b.close()
    assert all(torch.isfinite(dc.U[:, 4:-4, 4:-4, 4:-4]).all() for dc in dcs)
