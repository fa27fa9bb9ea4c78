"""Default launch shapes with 8 or 16 lanes per move: the moves in flight of at most 12 warps
per SM, which the pooled voxel table serves."""
import pytest
import torch

from chromo_gb300 import _native as nat

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lanes", [8, 16])
@pytest.mark.parametrize("per_sm", [1, 2, 3])
def test_default_moves_in_flight(lanes, per_sm):
    R = per_sm * torch.cuda.get_device_properties(0).multi_processor_count
    sim = nat.Sim([40] * R, [(4, 4, 4)] * R, 1, lanes_per_move=lanes)
    warps, g, moves, _ = sim.launch_shape()
    sim.close()
    assert g == lanes and moves == warps * (32 // lanes) <= 32
    assert warps * per_sm <= 12
