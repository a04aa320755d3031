"""Which input shapes ResNet50Int8.forward replays from a graph, without a GPU: the policy alone."""
import pytest

from glow_b200.resnet import Replays


def drive(calls):
    """The captures that a sequence of shapes leads to, and the most graphs held at a time."""
    r, captured, most = Replays(), [], 0
    for i, shape in enumerate(calls):
        if r.find(shape) is None and r.earned(shape):
            r.make_room()
            r.keep(shape, i)
            captured.append((i, shape))
        most = max(most, len(r.graphs))
    return captured, most, r


def test_a_shape_is_captured_once():
    assert drive(["a"] * 50)[0] == [(1, "a")]


@pytest.mark.parametrize("shapes", [2, 3, 4])
def test_shapes_that_alternate_keep_their_graphs(shapes):
    captured, most, _ = drive([i % shapes for i in range(100 * shapes)])
    assert [c[1] for c in captured] == list(range(shapes)) and most == shapes


@pytest.mark.parametrize("shapes,times", [(5, 1), (6, 2), (40, 1), (200, 2)])
def test_more_shapes_than_graphs(shapes, times):
    """Taken in turn, or each a few times in a row: captures stay rare, and what is held stays bounded."""
    calls = [i // times % shapes for i in range(4000)]
    captured, most, r = drive(calls)
    assert most <= Replays.KEPT and len(r.calls) <= Replays.REMEMBERED
    assert len(captured) <= Replays.KEPT + len(calls) // Replays.PATIENCE


def test_a_shape_that_came_to_stay_gets_its_graph():
    captured, _, r = drive(list("aabbccdd") + ["e"] * 40)
    assert captured[-1][1] == "e" and "a" not in r.graphs and r.find("e") is not None
