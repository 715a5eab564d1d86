"""Creating a plant waits for its own work only: not for another stream's kernels."""
import numpy as np
import pytest
import torch

import csdecomp_b200 as csd
from csdecomp_b200 import scenes

pytestmark = pytest.mark.gpu


def test_creation_does_not_wait_for_other_streams():
    sc = scenes.edge_check_scene()
    q = sc.random_configs(500, 1)
    ref = csd.CheckCollisionFreeCuda(q.T, sc.plant)  # everything loaded
    del sc.plant._csd_handle
    stream, done = torch.cuda.Stream(), torch.cuda.Event()
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        torch.cuda._sleep(1 << 30)  # about half a second
        done.record()
    h = csd.plant_handle(sc.plant)
    assert not done.query()
    torch.cuda.synchronize()
    assert h.dim == 7
    np.testing.assert_array_equal(csd.CheckCollisionFreeCuda(q.T, sc.plant), ref)
