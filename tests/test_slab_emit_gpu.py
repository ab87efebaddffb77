"""pf_slab_finish at capacities around a thread's 16 slots, a block's 4096 and a
step of its columns, slots none, some and all occupied, occupancy bytes on and
off a 16-byte boundary, wide and narrow values, every byte compared and the
outputs' rows past the count left alone."""
import ctypes

import numpy as np
import pytest
import torch

from pageflow_b200 import _native as N
from pageflow_b200.aggregation_slab import _DT

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cap", [1, 15, 16, 17, 1023, 4095, 4096, 4097, 50_001])
@pytest.mark.parametrize("keep,off", [(0.0, 0), (0.3, 0), (1.0, 0), (0.5, 3)])
def test_finish(cap, keep, off):
    rng = np.random.default_rng(cap)
    occ_np = (rng.random(cap) < keep).astype(np.uint8) * 255
    occ = torch.zeros(cap + off, dtype=torch.uint8, device="cuda")[off:]
    occ.copy_(torch.from_numpy(occ_np))
    vals = [torch.from_numpy(rng.integers(-1 << 62, 1 << 62, (cap, 3))).cuda(),
            torch.from_numpy(rng.integers(-1 << 30, 1 << 30, cap).astype(np.int32)).cuda(),
            torch.from_numpy(rng.standard_normal(cap)).cuda()]
    outs = [torch.full_like(v, -7) for v in vals]
    keys = torch.full((cap,), -7, dtype=torch.int64, device="cuda")
    host = torch.zeros(2, dtype=torch.int64, pin_memory=True)
    L = N.lib()
    ws = N.workspace(L.pf_slab_finish_workspace(cap), occ.device)
    dt = N.arr(ctypes.c_int, [_DT[v.dtype] for v in vals])
    N.check(L.pf_slab_finish(occ.data_ptr(), 100, cap, 3, N.arr(N._vp, [v.data_ptr() for v in vals]),
                             dt, N.arr(ctypes.c_int, [3, 1, 1]), keys.data_ptr(),
                             N.arr(N._vp, [o.data_ptr() for o in outs]), host.data_ptr(),
                             ws.data_ptr(), ws.numel(), N.stream_of(occ.device)), "finish")
    torch.cuda.synchronize()
    at = np.nonzero(occ_np)[0]
    n = int(host[0])
    assert n == len(at)
    assert np.array_equal(keys[:n].cpu().numpy(), at + 100)
    for o, v in zip(outs, vals):
        assert torch.equal(o[:n].cpu(), v.cpu()[at])
        assert bool((o[n:] == -7).all())
