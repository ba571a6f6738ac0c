"""The device time of an execution (AgoGraphPerfInternalInfo::kernel_wait): positive, no longer than the
CUDA events around the launch, and equal to them but for what launching a graph takes."""
import pytest

from mivisionx_b200 import vx as V
from mivisionx_b200 import workloads as WL

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("flags", [None, 0x20000])         # captured (clock readings inside), uncaptured (events)
@pytest.mark.parametrize("n,w,h", [(1, 320, 240), (4, 3840, 2160)])
def test_device_time_against_events(cuda, n, w, h, flags):
    import torch
    api = V.OpenVX()
    ctx = api.obj(api.vxCreateContext(), "context")
    g = WL.Cfg2Graph(api, ctx, [(w, h)] * n, flags=flags)
    g.run([WL.cfg2_scene(seed=3, width=w, height=h)] * n)
    stream = torch.cuda.ExternalStream(api.node_stream(g.node))
    got = []
    for _ in range(8):
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record(stream)
        api.ok(api.vxScheduleGraph(g.graph), "schedule")
        e1.record(stream)
        api.ok(api.vxWaitGraph(g.graph), "wait")
        e1.synchronize()
        got.append((api.gpu_ms_last(g.graph), e0.elapsed_time(e1)))
    for ms, events in got:
        assert 0 < ms <= events + 0.005                    # both clocks step by well under 5 us
    ms, events = min(got, key=lambda p: p[1] - p[0])
    assert events - ms <= 0.05                             # starting a graph costs some 10 us
