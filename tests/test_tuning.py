"""The fast calls' launch shapes and tuning: what the getters give can be set again, the defaults leave the choice to
the call, and the autotuner keeps what it does not tune."""
import json

import numpy as np
import pytest

from plainmp_gb300 import autotune, scenes
from plainmp_gb300 import workloads as W


def _chain():
    return scenes.make_constraint(W.chain7_robot(), W.chain7_scene())[1]


def test_every_tile_and_shape_is_given_back():
    cst = _chain()
    for tile in (0, 1, 2, 4, 8, 16, 32):
        for edge in autotune.EDGE_SHAPES:
            cst.set_fast_tuning(tile, 3, *edge)
            assert cst.get_fast_tuning() == (tile, 3, *edge)
    for shape in autotune.SHAPES:
        cst.set_fast_launch(*shape)
        assert cst.get_fast_launch() == shape


def test_tiles_to_try():
    """The least tile of a shape by its value (0 leaves the choice to the call), each once."""
    for cpb, _ in autotune.SHAPES:
        tiles = autotune.sphere_tiles(cpb)
        assert tiles[0] == max(1, 32 // cpb) and tiles[-1] == 32 and len(set(tiles)) == len(tiles) and 0 not in tiles
    assert (8, 256) in autotune.SHAPES
    assert autotune.SHAPES[0] == _chain().get_fast_launch() and autotune.EDGE_SHAPES[0] == _chain().get_fast_tuning()[2:]


@pytest.mark.gpu
def test_setting_what_was_read_keeps_the_calls_choice(tmp_path, monkeypatch):
    import torch
    from test_default_shape_gpu import shape_of

    from plainmp_gb300 import BoxMotionValidator

    monkeypatch.setenv("PMGPU_AUTOTUNE_CACHE", str(tmp_path / "a.json"))
    cst = _chain()
    v = BoxMotionValidator(cst, [0.05] * 7)
    Q = torch.from_numpy(W.chain7_configs(500)).cuda()
    S1, S2 = (torch.from_numpy(x).cuda() for x in W.chain7_edges(64))
    both = lambda: (shape_of(lambda: cst.is_valid_fast(Q), "k_fast_valid"),  # noqa: E731
                    shape_of(lambda: v.check_motion_fast(S1, S2), "k_fast_edges"))
    picked = both()
    assert picked == ((8, 256), (16, 128))
    launch, tuning = cst.get_fast_launch(), cst.get_fast_tuning()
    cst.set_fast_launch(64, 256)
    cst.set_fast_tuning(1, 4, 64, 256)
    assert both() == ((64, 256), (64, 256))
    cst.set_fast_launch(*launch)
    cst.set_fast_tuning(*tuning)
    assert both() == picked
    # tuning states leaves the edges alone, and the other way round
    shape, times = autotune.autotune(cst, Q, reps=3)
    assert times[min(times, key=times.get)] <= times["32x256/st0"] and "8x256/st8" in times
    assert shape_of(lambda: v.check_motion_fast(S1, S2), "k_fast_edges") == picked[1]
    states = cst.get_fast_launch(), cst.get_fast_tuning()[:2]
    autotune.autotune_edges(v, S1, S2, reps=3)
    assert (cst.get_fast_launch(), cst.get_fast_tuning()[:2]) == states
    # entries of other kernels' choices are not applied
    key = autotune.signature(cst, len(Q), False)
    assert key in json.loads((tmp_path / "a.json").read_text()) and key.endswith(f"|k{autotune.KERNELS}")
    assert np.array_equal(cst.is_valid_fast(Q).cpu().numpy(), cst.is_valid_batch(Q).cpu().numpy())
