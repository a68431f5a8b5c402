"""What the ops and tables promise beyond their values: inputs that are refused, layouts and types that are accepted, when a gradient
is reported as ready, what user hooks see, and what is held in memory between and during the passes."""
import numpy as np
import pytest
import torch

from vlm_training_b200 import ops

DEV = "cuda"
gpu = pytest.mark.gpu


def _rand(*shape, scale=1.0, seed=0, dtype=torch.bfloat16):
    return (torch.randn(*shape, generator=torch.Generator().manual_seed(seed + sum(shape))) * scale).to(DEV, dtype)


# sides off the merge size, smaller than it, negative: refused on the host before anything reaches the device
@pytest.mark.parametrize("device", ["cpu", "cuda"])
@pytest.mark.parametrize("grids", [[[1, 2, 3]], [[1, 3, 2]], [[1, 1, 1]], [[1, 28, 37]], [[1, 27, 36]], [[1, 4, 4], [1, 1, 4]], [[1, -2, -2]]])
def test_image_sizes_off_the_merge_size_are_refused(grids, device):
    from vlm_training_b200.models.config import VisionConfig
    from vlm_training_b200.models.vision import VisionPlan

    with pytest.raises(ValueError):
        VisionPlan.build(grids, VisionConfig(hidden_size=64, num_heads=2, num_position_embeddings=2304, spatial_merge_size=2), device)


@gpu
def test_position_indices_stay_in_the_table():
    """The plan kernel clamps its coordinates to the tables, whatever the image sizes say."""
    images = torch.tensor([[1, 3, 37, 0], [1, 2, 1, 111]], dtype=torch.int32, device=DEV)
    trig = torch.ones(37 * 4 * 2, device=DEV)
    index = ops.vision_plan(images, trig, 4, 48, 2, 113)[2]
    assert int(index.min()) >= 0 and int(index.max()) < 48 * 48
