"""New intrinsics do not reach into work that was started with the old ones."""
import numpy as np
import pytest
import torch

import synth
from superscanner_gb300 import GPUVoxelGrid

pytestmark = pytest.mark.gpu

ROWS, COLS = 97, 131
INTR, OTHER = (107.0, 108.0, 65.0, 48.0), (90.0, 91.5, 60.0, 50.0)


def _scene(n):
    sc = synth.Scene(2, 1234)
    P = sc.trajectory(n, 42)
    depth, _ = sc.render(P, ROWS, COLS, INTR, noise=True, noise_seed=7, color=False)
    return P, [torch.from_numpy(d.view(np.int16)).cuda() for d in depth]


def _grid(storage="f32"):
    g = GPUVoxelGrid(int(1e9), 0.032, 0.008, ROWS, COLS, storage=storage, with_color=False, hash_buckets=1 << 16,
                     max_weight=255)
    g.setIntrinsic(*INTR)
    return g


@pytest.mark.parametrize("exact", [True, False])
def test_new_intrinsics_wait_for_calls_in_flight(exact):
    """On a stream that the default stream does not wait for, behind work that holds it up for a tenth of a second."""
    P, dev = _scene(1)
    E = P[0].astype(np.float32)
    out = []
    for change in (False, True):
        g = _grid()
        torch.cuda.synchronize()
        side = torch.cuda.Stream()
        with torch.cuda.stream(side):
            torch.cuda._sleep(200_000_000)
            if exact:
                g.integrate(None, dev[0], E, withColor=False)
            else:
                g.integrate_fast(dev[0], E)
        if change:
            g.setIntrinsic(*OTHER)
        g.sync(side)
        out.append(g.export_blocks(with_color=False))
        g.close()
    for k in ("keys", "coords", "sdf", "w"):
        assert np.array_equal(out[0][k], out[1][k])


@pytest.mark.parametrize("exact", [True, False])
def test_a_captured_frame_takes_new_intrinsics(exact):
    """The per-frame graph, captured before the intrinsics changed, against frames launched one by one."""
    from superscanner_gb300.pipeline import Pipeline
    P, dev = _scene(6)
    out = []
    for graph in (False, True):
        g = _grid("f16")
        pipe = Pipeline(g, use_graph=graph, persistent_track=False, exact_fusion=exact)
        pipe.set_pose(P[0])
        pipe.frame(dev[0], track=False)
        pipe.frame(dev[1])
        pipe.frame(dev[2])
        torch.cuda.synchronize()
        g.setIntrinsic(*OTHER)
        poses = []
        for k in (3, 4, 5):
            pipe.frame(dev[k])
            poses.append(pipe.pose())
        maps = pipe.maps_tensors()
        g.sync()
        out.append((np.stack(poses), *(m.cpu().numpy() for m in maps), *g.export_blocks(with_color=False).values()))
        pipe.close()
        g.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b) if a is not None else b is None
