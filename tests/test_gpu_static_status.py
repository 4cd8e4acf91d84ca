"""The allocation-free forces' status word: an error that a call found belongs to that
call, also when its second kernel is refused by the runtime."""
import ctypes

import numpy as np
import pytest

from test_zz_no_alloc import INDEX, _args, _entry, _upload

pytestmark = pytest.mark.gpu


def test_status_of_a_call_that_fails_to_launch(gpu_lib):
    import torch
    L, fn = gpu_lib, _entry(gpu_lib)
    g = L.Domain(L.LuleshProblem(nx=3, keep_aux=True))
    L.run(g, 5)
    dev = {n: torch.from_numpy(g.field(n)).cuda() for n in INDEX}
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    site = ctypes.c_int32()
    v = np.array(g.field("v"))
    v[4] = -1.0
    _upload(g, dev, {"v": v})
    a = _args(L, g, dev, 0)
    torch.cuda.synchronize()
    volume_error = fn(ctypes.byref(a), stream, ctypes.byref(site))
    assert volume_error != 0 and site.value != 0
    # 2^40 nodes: 2^32 blocks, which the runtime refuses before anything runs
    a.num_node = 2 ** 40
    refused = fn(ctypes.byref(a), stream, ctypes.byref(site))
    assert refused not in (0, volume_error) and site.value == 0
    _upload(g, dev)
    a = _args(L, g, dev, 0)
    torch.cuda.synchronize()
    assert fn(ctypes.byref(a), stream, ctypes.byref(site)) == 0 and site.value == 0
    assert np.isfinite(dev["fx"].cpu().numpy()).all()
