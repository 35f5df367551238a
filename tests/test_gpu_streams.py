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
