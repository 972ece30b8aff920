"""GPU check that a context whose first build found little free memory uses the memory once it is free.

Chunks show in the number of launches; the results agree to rounding (other split factors), within the repository's
parity tolerance of 1e-10."""
import numpy as np
import pytest

from green_gpu_b200 import native, synth

pytestmark = pytest.mark.gpu


def test_plan_grows_when_memory_is_free_again():
    import torch
    s = synth.make_system(mesh=(2, 2, 1), nao=6, NQ=480, ns=1, beta=10.0, lam=100.0, nts=24, nw_b=21, seed=1)
    ctx, other = native.context_for(s), native.context_for(s)
    try:
        ref = other.gw_sigma(s.G_tskij)
        whole = other.launch_count()
        other.close()
        torch.cuda.synchronize()
        free, _ = torch.cuda.mem_get_info()
        hold = torch.empty(free - (1000 << 20), dtype=torch.uint8, device="cuda")  # the build takes 1.5 GB
        first = ctx.gw_sigma(s.G_tskij)
        assert ctx.launch_count() > whole
        del hold
        torch.cuda.empty_cache()
        second = ctx.gw_sigma(s.G_tskij)
        assert ctx.launch_count() == whole
    finally:
        other.close()
        ctx.close()
    for out in (first, second):
        assert np.abs(out - ref).max() < 1e-10 * np.abs(ref).max()
