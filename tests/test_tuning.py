"""The fast calls' launch shapes and tuning: what the getters give can be set again."""
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
