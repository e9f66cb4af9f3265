"""Device memory of a handle: the list of deferred HLLD faces must not need
memory of its own, so that what fits with another Riemann solver fits with
HLLD."""
import pytest

from cumc3d_b200 import engine, models

pytestmark = pytest.mark.gpu


def test_hlld_handle_needs_no_more_memory_than_hllc():
    import torch
    used = {}
    for rs in ("hllc", "hlld", "hllc", "hlld"):   # the first pair also loads the kernels
        spec, _, _ = models.blast_3d(96, nx=96, ny=80, nz=72, riemann=rs)
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        s = engine.Solver(spec)
        s.sync()
        used[rs] = before - torch.cuda.mem_get_info()[0]
        s.close()
    assert abs(used["hlld"] - used["hllc"]) <= 4 << 20, used   # two allocation granules
