"""Downloads into page-locked and partly page-locked memory."""
import numpy as np
import pytest
import torch

import bfx
from bfx import workloads

pytestmark = pytest.mark.gpu


def label_image(ws, batch, bits, pred):
    bfx._check(bfx.load().bfx_download_labels(ws._h, bfx.u32(batch), bfx._ptr(bits), bfx._ptr(pred)))


@pytest.mark.parametrize("locked", ["all", "first half", "second half"])
def test_page_locked_outputs(gpu, locked):
    layout, grid = workloads.build_graph("c1")
    desc = bfx.make_description(layout, workloads.full_graph_queries(layout, grid, 8, 3), 8)
    resident = bfx.ResidentDeviceGraph.upload_once(layout)
    ws = bfx.Workspace(resident)
    ws.prepare([desc])
    ws.execute(bfx.GpuRunOptions())
    bits, pred = ws.download_labels(0, 8)
    n = bits.size
    if locked == "all":
        host = torch.full((2, n), -2, dtype=torch.int32, pin_memory=True)
        got = host.numpy().view(np.uint32)
        label_image(ws, 0, got[0], got[1])
    else:
        page = 4096
        raw = np.full(2 * n + 2 * page, 0xFFFFFFFE, np.uint32)
        start = (-raw.ctypes.data // 4) % (page // 4)
        got = raw[start:start + 2 * n].reshape(2, n)
        assert got.ctypes.data % page == 0 and n * 4 % (2 * page) == 0
        at = got.ctypes.data + (0 if locked == "first half" else n * 2)
        cudart = torch.cuda.cudart()
        assert int(cudart.cudaHostRegister(at, n * 2, 0)) == 0  # half of the first output
        label_image(ws, 0, got[0], got[1])
        assert int(cudart.cudaHostUnregister(at)) == 0
    np.testing.assert_array_equal(got[0].reshape(bits.shape), bits)
    np.testing.assert_array_equal(got[1].reshape(pred.shape), pred)
    ws.close()
    resident.close()
