"""How often certify_map makes the host wait: once where the first stage proves every cell, three times without the
preproof (the first stage's counts, the fallback's jobs, the record)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,waits", [("PrescreenCertificateConfig", 1), ("AdaptiveCertificateConfig", 3)])
def test_waits(kind, waits):
    from torch.profiler import ProfilerActivity, profile
    from seq_vp_3d_b200 import certificate as cert
    from seq_vp_3d_b200.grid import grid_from_shape
    shape = (12, 14, 18)
    u = np.zeros(shape + (3,))
    u[1:-1, 1:-1, 1:-1] = np.random.default_rng(0).uniform(-.05, .05, (10, 12, 16, 3))
    grid, config, ud = grid_from_shape(shape, (1., 1., 1.)), getattr(cert, kind)(delta=0.), torch.from_numpy(u).cuda()
    run = lambda: cert.certify_map(ud, grid, config=config, with_hash=False)
    assert run().status == "certified_feasible"
    with profile(activities=[ProfilerActivity.CUDA, ProfilerActivity.CPU]) as p:
        run()
    assert sum(e.name == "cudaStreamSynchronize" for e in p.events()) == waits
