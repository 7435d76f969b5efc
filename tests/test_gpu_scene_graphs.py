"""A scene and a batch give back every graph that they have made: as many destroyed as instantiated."""
import pytest

from metakonga_gb300 import engine

from .cases import packed_scene
from .cuda_calls import runtime_calls

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch", [False, True])
@pytest.mark.parametrize("calls", [(1,), (20,), (20, 1)])
def test_graphs_given_back(cuda, calls, batch):
    def work():
        scenes = [engine.DeviceScene(packed_scene(n_side=4), mode=engine.MODE_MIXED) for _ in range(2 if batch else 1)]
        b = engine.Batch(scenes) if batch else scenes[0]
        for n in calls:
            b.step(n, check=True)
        if batch:
            b.close()
        for d in scenes:
            d.close()

    names = runtime_calls(work)
    made = sum("GraphInstantiate" in x for x in names)
    assert made > 0 and made == sum("GraphExecDestroy" in x for x in names), names
