"""One scene and callers' streams, on the GPU.  Streams of torch do not wait
for the legacy stream (cudaStreamNonBlocking), nor it for them.

Bars (written here): the same rays in another order of float additions, so
flux images within L1 1e-5 and FP64 powers within 1e-9 relative.
"""
import numpy as np
import pytest

import solarenergy_chier_b200 as q
from solarenergy_chier_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def small(tmp_path_factory, cuda_device):
    """50 heliostats, 655 M rays a trace: several milliseconds on the device."""
    return synth.small_field(tmp_path_factory.mktemp("streams"), seed=4, groups=4)


def assert_same(img, want, bar=1e-5):
    assert want.sum() > 0 and np.abs(img.astype(np.float64) - want).sum() <= bar * want.sum(dtype=np.float64)


@pytest.mark.parametrize("change", ["set_sample_pool", "generate_sample_pool", "set_sun"])
def test_a_change_waits_for_traces_of_other_streams(change, small):
    """New pools or a new sun while a trace of another stream runs: the trace
    keeps the samples and the walk codes that it started with."""
    import torch

    s = q.Scene(small.scene, small.config, device=0, seed=2)
    ids = list(range(s.num_heliostats))
    s.generate_sample_pool(3)
    s.trace(ids)
    want, power = s.image(0), s.power()[0]
    wide = q.Scene(small.scene, small.config, device=0, seed=9)
    wide.generate_sample_pool(8, q.SUNSHAPE_PILLBOX, 0.02)
    pools = wide.get_sample_pool()
    s.clear()
    s.clear_power()
    torch.cuda.synchronize()
    stream = torch.cuda.Stream()
    s.trace(ids, stream=stream.cuda_stream)
    if change == "set_sample_pool":
        s.set_sample_pool(*pools)
    elif change == "generate_sample_pool":
        s.generate_sample_pool(8, q.SUNSHAPE_PILLBOX, 0.02)
    else:
        s.set_sun(synth.sun_direction(110.0, 25.0))
    torch.cuda.synchronize()
    assert_same(s.image(0), want)
    np.testing.assert_allclose(s.power()[0], power, rtol=1e-9, atol=0)


def test_a_captured_call_of_one_heliostat(small):
    """One-heliostat traces captured right after the light range changed, then
    replayed after traces of other ranges and lists: the graph depends on no
    memory of the capturing call."""
    import torch

    s = q.Scene(small.scene, small.config, device=0, seed=2)
    s.trace([3])  # another light range before
    s.set_light_range(5, 42)
    s.clear()
    s.trace([3])
    s.trace([7])
    want, power = s.image(0), s.power()[0]
    s.set_light_range(0, 200)
    s.trace([3])
    s.set_light_range(5, 42)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        stream = torch.cuda.current_stream()
        s.trace([3], stream=stream)
        s.trace([7], stream=stream)
    s.set_light_range(0, 300)
    s.trace([9])
    s.trace([1, 4, 6])
    for _ in range(2):
        s.clear()
        s.clear_power()
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        assert_same(s.image(0), want)
    assert s.power()[0][7] == pytest.approx(power[7], rel=1e-12)


def test_calls_of_one_heliostat_on_several_streams(small):
    """Calls of different light counts and chunk sizes follow one another on
    three streams without waiting: the image is that of the calls in turn."""
    import torch

    s = q.Scene(small.scene, small.config, device=0, seed=2)
    calls = [(h, lights) for h in range(12) for lights in (16, 2048, 600)]  # 8-, 16- and 8-iteration chunks
    s.trace(list(range(s.num_heliostats)))  # the power partials' buffer is large enough from here on

    def traced(streams):
        s.clear()
        torch.cuda.synchronize()
        for k, (h, lights) in enumerate(calls):
            s.set_light_range(0, lights)
            s.trace([h], stream=streams[k % len(streams)])
        torch.cuda.synchronize()
        return s.image(0)

    want = traced([torch.cuda.current_stream()])
    assert_same(traced([torch.cuda.Stream() for _ in range(3)]), want)


def test_images_keep_their_values_while_another_stream_traces(small):
    """Copies of an image taken while another stream traces onto it hold at
    least what earlier traces left: deposits only add."""
    import torch

    from solarenergy_chier_b200 import shard

    s = q.Scene(small.scene, small.config, device=0, seed=2)
    ids = list(range(s.num_heliostats))
    s.trace(ids)
    want = torch.from_numpy(s.image(0))
    view = shard.device_image_tensor(s, 0)
    tracing, reading = torch.cuda.Stream(), torch.cuda.Stream()
    copies = [torch.empty_like(want).pin_memory() for _ in range(8)]
    with torch.cuda.stream(reading):
        copies[0].copy_(view, non_blocking=True)
    torch.cuda.synchronize()
    for _ in range(6):
        s.trace(ids, stream=tracing)
    during = 0
    with torch.cuda.stream(reading):
        for c in copies:
            c.copy_(view, non_blocking=True)
            reading.synchronize()
            during += not tracing.query()
    torch.cuda.synchronize()
    assert during > 0, "no copy was taken during the traces"
    for c in copies:
        assert float((want - c).clamp(min=0).sum()) <= 1e-6 * float(want.sum())
    assert_same(s.image(0), 7.0 * want.numpy())


def test_a_waited_trace_is_in_the_image_whatever_other_streams_do(small):
    """One list traced on two streams: after waiting for one of them alone,
    the image holds that trace."""
    import torch

    from solarenergy_chier_b200 import shard

    s = q.Scene(small.scene, small.config, device=0, seed=2)
    ids = list(range(s.num_heliostats))
    s.trace(ids)
    want = torch.from_numpy(s.image(0))
    view = shard.device_image_tensor(s, 0)
    got = torch.empty_like(want).pin_memory()
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    for first, second in ((a, b), (b, a), (a, b)):
        s.clear()
        torch.cuda.synchronize()
        s.trace(ids, stream=first)
        s.trace(ids, stream=second)
        with torch.cuda.stream(first):
            got.copy_(view, non_blocking=True)
            first.synchronize()
        assert float((want - got).clamp(min=0).sum()) <= 1e-5 * float(want.sum())
        torch.cuda.synchronize()
