"""A context's zero fills are done before its first kernels, whatever the
caller has queued on the default stream (another library's kernels)."""
import numpy as np
import pytest

from komegafoulingmodel_b200 import Lattice, desc_default
from komegafoulingmodel_b200 import geometry as G


@pytest.mark.gpu
def test_geometry_and_state_with_a_busy_default_stream():
    import torch
    nx, ny = 256, 66
    h = 8.0 * 0.5 * (1 - np.cos(2 * np.pi * np.arange(nx) / 128))
    ch = G.channel_from_walls(nx, ny, 0.5 + h, ny - 1.5 - h, wall_distance=False)
    f = G.equilibrium_state(ch, ux=0.01)
    pinned = torch.from_numpy(f).pin_memory().numpy()
    d = desc_default()
    d.nx, d.nx_full, d.ny, d.tau, d.fterm, d.mu = nx, nx, ny, 1.25, 1e-6, 0.1
    a = torch.randn(8192, 8192, device="cuda")
    (a @ a).sum().item()  # the library's own set-up is not part of the queue
    for _ in range(40):   # tens of milliseconds on the default stream
        a = (a @ a) * 1e-4
    with Lattice(d) as L:
        L.set_walls(0.5 + h, ny - 1.5 - h)
        geo = L.get_geometry()
        L.set_state(pinned)
        g = L.get_state()[0]
    torch.cuda.synchronize()
    assert np.array_equal(geo["ntype"], ch.ntype)
    assert np.array_equal(geo["ibb_idx"], ch.ibb_idx)
    fl = np.tile(ch.fluid_mask().ravel(), 9)
    assert np.abs(g - f)[fl].max() < 1e-7
