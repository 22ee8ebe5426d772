"""The wide tree that the device builds at upload (csrc/wide_build.cu) against the host's build of it: which trees qualify, and
how many nodes they have. A film alone does not tell: a tree that is turned down renders the same bits in preorder."""
import numpy as np
import pytest

from test_ordered_traversal import CHAINS, _arrays, _broken, _chain


def _host_nodes(wfb, scene):
    return scene.test_traverse_ordered(np.zeros(0, wfb.RAY))[1]["tree"]


# a chain's wide tree has a level per 3 leaves: these lie either side of the 96 levels that a tree may have
EDGE_CHAINS = list(range(286, 296))


def test_host_build_has_the_level_limit(wfb):
    nodes = [_host_nodes(wfb, wfb.Scene.from_arrays(_chain(wfb, n, False))) for n in EDGE_CHAINS]
    qualifies = [n > 0 for n in nodes]
    assert qualifies == sorted(qualifies, reverse=True) and qualifies[0] and not qualifies[-1]
    assert max(nodes) == 96  # one node per level
    assert _host_nodes(wfb, wfb.Scene.from_arrays(_chain(wfb, 400, True))) == 0


@pytest.mark.gpu
@pytest.mark.parametrize("n", [n for n, _ in CHAINS] + EDGE_CHAINS)
def test_chains_on_the_device(wfb, n):
    scene = wfb.Scene.from_arrays(_chain(wfb, n, False))
    assert scene.wide_nodes() == _host_nodes(wfb, scene)


# one block in shared memory (to 1,024 preorder nodes), the first levels in one launch, and levels in launches of their own
@pytest.mark.gpu
@pytest.mark.parametrize("name", ["one_leaf", "cornell36", "balls", "icospheres", "heightfield"])
def test_scenes_on_the_device(wfb, name):
    scene = wfb.Scene.from_arrays(_arrays(wfb, name))
    nodes = scene.wide_nodes()
    assert nodes > 0 and nodes == _host_nodes(wfb, scene)


@pytest.mark.gpu
@pytest.mark.parametrize("how", ["grown", "shrunk", "shared"])
@pytest.mark.parametrize("name", ["balls", "icospheres"])
def test_trees_that_do_not_qualify_on_the_device(wfb, name, how):
    scene = wfb.Scene.from_arrays(_broken(_arrays(wfb, name), how))
    assert scene.wide_nodes() == _host_nodes(wfb, scene) == 0
