"""A matrix-free assembly that fails gives its stream back: a stream that is
lost keeps half a megabyte of device memory."""
import pytest

from fasterhenry_b200 import fixtures as F

pytestmark = pytest.mark.gpu


def test_failed_assemblies_keep_no_device_memory(fh):
    import torch
    deck = F.meander_legs(4, nw=2, nh=2)
    geometry = fh.Geometry.from_deck(deck)
    too_fine = fh.IterativeParams(pfft=fh.PfftParams(spacing=1e-7))

    def fail(times):
        for _ in range(times):
            with pytest.raises(fh.FasterHenryError) as e:
                fh.IterativeSystem.assemble(geometry, deck.ports, deck.discretization, too_fine)
            assert "padded points" in str(e.value)

    fail(10)
    before = torch.cuda.mem_get_info()[0]
    fail(200)
    assert before - torch.cuda.mem_get_info()[0] < 16 << 20
    with fh.IterativeSystem.assemble(geometry, deck.ports, deck.discretization) as s:
        s.impedance(1e9)
