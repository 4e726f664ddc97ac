"""GPU: the persistent CTAs that a batch reports are those of the scatter it
launches: with tap lists the tap lanes', else those of the kernel that evaluates
the taps."""
import pytest

from conftest import load_case


@pytest.mark.gpu
# a 2048-entry table: 16 bytes an entry (124 KB a CTA, one per SM) where the taps are
# evaluated, 4 in the tap lanes (111 KB, two per SM)
@pytest.mark.parametrize("tap_lists,per_sm", [(True, 2), (False, 1)])
def test_batch_reports_its_scatter(oracle, tap_lists, per_sm):
    import torch

    from fastrecon_gb300 import batch as fb
    c = load_case("radial2d_small")
    b = fb.GridBatch(2, c["G"], c["W"], lut=oracle.kb_lut(c["W"], 2.0, 2048), tile=(32, 16, 0), coil_group=16,
                     tap_lists=tap_lists)
    b.set_trajectories(torch.from_numpy(c["traj"]).cuda(), [c["traj"].shape[0]])
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert b.stats()["ctas"] == per_sm * sms
