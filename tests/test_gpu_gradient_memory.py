"""The gradient's memory check counts what the library's cache holds idle: its
buffers come from there, so a large system or operator that has been closed
does not get it refused.  The rest of the device is taken by another
allocator meanwhile."""
import numpy as np
import pytest

from fasterhenry_b200 import fixtures as F

pytestmark = pytest.mark.gpu


def test_idle_cached_memory_counts_as_free(fh):
    import torch
    deck = F.meander_legs(40, nw=10, nh=2)
    params = [fh.Param("width", 0), fh.Param("x", 1)]
    hog = None
    with fh.MeshSystem.assemble(fh.Geometry.from_deck(deck), deck.ports, deck.discretization) as s:
        n = len(s.filaments())
        need = 48 * n * n  # six derivative matrices
        want = s.gradient(1e8, params)
        try:
            # 2 GB for the spectrum of a torus, idle afterwards
            fh.grid_convolution(np.ones((1, 2, 2, 20)), (1200, 1200, 40), 1e-3)
            torch.cuda.synchronize()
            hog = torch.empty(torch.cuda.mem_get_info()[0] - (48 << 20), dtype=torch.uint8, device="cuda")
            assert torch.cuda.mem_get_info()[0] < need / 2
            got = s.gradient(1e8, params)
        finally:
            del hog
            torch.cuda.empty_cache()
            fh.release_cached_memory()
    assert np.array_equal(got.impedance_ohm, want.impedance_ohm)
    assert np.max(np.abs(got.gradient - want.gradient)) <= 1e-12 * np.max(np.abs(want.gradient))
