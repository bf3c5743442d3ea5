"""The chain's kernels against the oracle, byte for byte, where their fast and
general paths meet: parameters outside the fast E-step's range and histograms
at the ends of the bin range, scorers and ROI statistics with infinities and
NaN, tied analogs, the smallest and largest chunks, traces and scales that
wrap int16."""
import numpy as np
import pytest

from hw_b200 import abi, workloads

import harness
import synth

pytestmark = pytest.mark.gpu


def _eq(name, a, b):
    ab, bb = (np.ascontiguousarray(x).view(np.uint8) for x in (a, b))
    assert ab.shape == bb.shape and not (ab != bb).any(), f"{name}: {int((ab != bb).sum())} bytes differ"


def _both(cfg, lanes, F, call):
    """call(backend) on the oracle and on the GPU: equal results, or the same
    reference assertion from both."""
    out = []
    for make in (harness.OracleBackend, harness.GpuBackend):
        try:
            out.append(tuple(call(make(cfg, lanes, F))))
        except RuntimeError as e:
            out.append([n for n in abi.STATUS_NAMES.values() if n in str(e)])
    if isinstance(out[0], list):
        assert out[0] == out[1]
        return
    for i, (a, b) in enumerate(zip(*out)):
        _eq(f"output {i}", a, b)


@pytest.mark.parametrize("F", [48, 512])
@pytest.mark.parametrize("pedestal,sensitivity,extreme", [(0, 1.0, False), (13, 1.9, False), (-32768, 0.01, True),
                                                          (32767, 62.0, True), (5, 100.0, True), (0, 3.0e7, False)])
def test_baseline_ranges(F, pedestal, sensitivity, extreme):
    lanes = 3
    cfg = workloads.chip_config()
    cfg.pedestal, cfg.photoelectron_sensitivity = pedestal, sensitivity
    chunks = 6 if F > 100 else 40
    tr = synth.traces(lanes, chunks * F, seed=F + pedestal % 97, walk_sigma=0.05)
    if extreme:
        tr[0, 3::11] = 32767
        tr[1, 5::13] = -32768

    def call(b):
        out = []
        for c in range(chunks):
            out += b.baseline(np.ascontiguousarray(tr[:, c * F:(c + 1) * F]), c * F)
        return out
    _both(cfg, lanes, F, call)
