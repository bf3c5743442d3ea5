"""The chain's kernels against the oracle, byte for byte, where their fast and
general paths meet: parameters outside the fast E-step's range and histograms
at the ends of the bin range, scorers and ROI statistics with infinities and
NaN, tied analogs, the smallest and largest chunks, traces and scales that
wrap int16."""
import numpy as np
import pytest

from hw_b200 import abi, workloads
from hw_b200.native import HwError

import harness
import synth

pytestmark = pytest.mark.gpu


def _eq(name, a, b):
    ab, bb = (np.ascontiguousarray(x).view(np.uint8) for x in (a, b))
    assert ab.shape == bb.shape and not (ab != bb).any(), f"{name}: {int((ab != bb).sum())} bytes differ"


def _both(cfg, lanes, F, call, error=None):
    """call(backend) on the oracle and on the GPU: equal results or, where
    `error` names a status, that reference assertion from both.  Any other
    failure is the test's."""
    oracle_backend, gpu = (make(cfg, lanes, F) for make in (harness.OracleBackend, harness.GpuBackend))
    if error:
        with pytest.raises(RuntimeError, match=f"^oracle: {error}: "):
            call(oracle_backend)
        with pytest.raises(HwError) as e:
            call(gpu)
        assert abi.STATUS_NAMES[e.value.code] == error
        return
    want, got = list(call(oracle_backend)), list(call(gpu))
    assert len(want) == len(got) > 0
    for i, (a, b) in enumerate(zip(want, got)):
        _eq(f"output {i}", a, b)


def _estimate_inputs(lanes):
    """Histogram, statistics and prior of a pool's first estimate (oracle)."""
    cfg = workloads.small_config()
    tr = synth.traces(lanes, 512 * 8, seed=5, gain_sigma=0.3, empty_fraction=0.2)
    pipe = harness.Pipeline(harness.OracleBackend(cfg, lanes, 512), cfg)
    for c in range(8):
        rec = pipe.process(np.ascontiguousarray(tr[:, c * 512:(c + 1) * 512]), c * 512)
        if "init_models" in rec:
            prior = rec["init_models"]
        if "hist" in rec:
            return cfg, rec["hist"], rec["agg"], prior
    raise AssertionError("no estimate")


@pytest.mark.parametrize("kind", ["plain", "one_bin", "ends", "far", "empty", "narrow", "inf_mean", "zero_var",
                                  "wide_bins", "bright"])
def test_estimate_paths(kind):
    lanes = 2
    cfg, hist, stats, prior = _estimate_inputs(lanes)
    hist, stats, prior = hist.copy(), stats.copy(), prior.copy()
    odd = slice(None, None, 3)          # ZMWs of every warp, not all of them
    bins = hist["bin_count"]
    if kind == "one_bin":
        bins[:, :, odd] = 0
        bins[:, 40, odd] = 4000
    elif kind == "ends":
        bins[:, 0, odd] = 7
        bins[:, 299, odd] = 5
    elif kind == "far":
        bins[:, 250:260, 5] = 1
    elif kind == "empty":
        bins[:, :, odd] = 0
    elif kind == "narrow":
        hist["bin_size"][:, odd] *= np.float32(1e-3)
    elif kind == "inf_mean":
        prior["analogs"]["means"][:, 1, odd] = 0x7c00
    elif kind == "zero_var":
        stats["baseline_stats"]["moment2"][:, odd] = 0.0
    elif kind == "wide_bins":
        hist["bin_size"][:, odd] *= np.float32(1e5)
    elif kind == "bright":
        prior["analogs"]["means"][:, :, odd] = abi.f32_to_f16(np.float32(6.0e4))
    _both(cfg, lanes, 512, lambda b: b.estimate(hist, stats, (0, 4096), (0, 512), prior),
          error="HW_ERR_NUMERIC" if kind == "inf_mean" else None)


def _models(lanes, seed=0):
    import oracle
    cfg = workloads.small_config()
    cfg.model_estimation_mode = abi.FIXED_ESTIMATIONS
    m = oracle.static_model(cfg, lanes)
    rng = np.random.default_rng(seed)
    for a, amp in enumerate(workloads.AMPLITUDES_DN):
        g = rng.lognormal(0.0, 0.2, (lanes, abi.LANE)).astype(np.float32)
        m["analogs"]["means"][:, a] = abi.f32_to_f16(amp * g)
        m["analogs"]["vars"][:, a] = abi.f32_to_f16(64.0 + 0.5 * amp * g + 0.01 * (amp * g) ** 2)
    m["baseline"]["means"] = abi.f32_to_f16(np.zeros((lanes, abi.LANE)))
    m["baseline"]["vars"] = abi.f32_to_f16(np.full((lanes, abi.LANE), 64.0))
    return m


@pytest.mark.parametrize("kind", ["plain", "equal_analogs", "below_baseline", "zero_var", "inf_var", "reversed_roi",
                                  "open_roi"])
@pytest.mark.parametrize("F", [48, 208, 1024])
def test_label_paths(kind, F):
    lanes = 3
    cfg = workloads.small_config()
    m = _models(lanes)
    odd = slice(1, None, 3)
    if kind == "equal_analogs":
        for f in ("means", "vars"):
            m["analogs"][f][:, 1:, odd] = m["analogs"][f][:, :1, odd]
    elif kind == "below_baseline":
        m["analogs"]["means"][:, 2, odd] = abi.f32_to_f16(np.float32(-30.0))
    elif kind == "zero_var":
        m["baseline"]["vars"][:, odd] = 0
        m["analogs"]["vars"][:, 0, odd] = 0
    elif kind == "inf_var":
        m["baseline"]["vars"][:, odd] = 0x7c00
        m["analogs"]["vars"][:, 3, odd] = 0x7c00
    elif kind == "reversed_roi":
        cfg.roi_upper_threshold, cfg.roi_lower_threshold = 2.0, 7.0
    elif kind == "open_roi":
        cfg.roi_upper_threshold = cfg.roi_lower_threshold = -1e9
    tr = synth.traces(lanes, 4 * F, seed=F, gain_sigma=0.2, empty_fraction=0.1, baseline=0.0)
    if kind == "plain":
        tr[0, ::97] = 32767
        tr[1, ::89] = -32768

    def call(b):
        out = []
        for c in range(4):
            out += b.label(np.ascontiguousarray(tr[:, c * F:(c + 1) * F]), m)
        return out
    _both(cfg, lanes, F, call)


@pytest.mark.parametrize("upper,lower", [(2.0, 0.0), (0.0, 0.0), (0.0, -0.0), (-0.0, 0.0), (0.0, 2.0)])
def test_label_zero_threshold(upper, lower):
    """ROI thresholds of 0 and an infinite baseline variance: the statistic is
    0 for a positive trace and -0 for a negative one, and both reach 0."""
    lanes, F = 2, 96
    cfg = workloads.small_config()
    cfg.roi_upper_threshold, cfg.roi_lower_threshold = upper, lower
    good, bad = _models(lanes), _models(lanes)
    bad["baseline"]["vars"][:, ::2] = 0x7c00
    tr = synth.traces(lanes, 6 * F, seed=1, gain_sigma=0.2, empty_fraction=0.1, baseline=0.0)
    tr[:, ::7] = 0

    def call(b):
        out = []
        for c in range(6):
            out += b.label(np.ascontiguousarray(tr[:, c * F:(c + 1) * F]), good if c % 2 else bad)
        return out
    _both(cfg, lanes, F, call)


@pytest.mark.parametrize("kind", ["zero_var", "zero_analog_var", "nan_var", "nan_mean", "inf_var"])
@pytest.mark.parametrize("F", [48, 512])
def test_label_model_recovers(kind, F):
    """A ZMW whose model scores NaN in one chunk and is ordinary in the next:
    the next chunk's latent frames still take the old model, and the NaN they
    leave in the log-likelihoods is the generic rows' to carry."""
    lanes = 2
    good, bad = _models(lanes), _models(lanes)
    odd = slice(1, None, 3)
    if kind == "zero_var":
        bad["baseline"]["vars"][:, odd] = 0
    elif kind == "zero_analog_var":
        bad["analogs"]["vars"][:, 0, odd] = 0
    elif kind == "nan_var":
        bad["analogs"]["vars"][:, 1, odd] = 0x7e00
    elif kind == "nan_mean":
        bad["analogs"]["means"][:, 2, odd] = 0x7e00
    elif kind == "inf_var":
        bad["baseline"]["vars"][:, odd] = 0x7c00
        bad["analogs"]["vars"][:, 3, odd] = 0x7c00
    tr = synth.traces(lanes, 6 * F, seed=F, gain_sigma=0.2, empty_fraction=0.1, baseline=0.0)

    def call(b):
        out = []
        for c in range(6):
            out += b.label(np.ascontiguousarray(tr[:, c * F:(c + 1) * F]), good if c % 2 else bad)
        return out
    _both(workloads.small_config(), lanes, F, call)


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


@pytest.mark.parametrize("encoding", [0, 1])
@pytest.mark.parametrize("lanes_per_pool,packet_blocks,width", [(16, 2, 128), (16, 1, 128), (2, 4, 64), (1, 4, 64),
                                                                (7, 64, 64), (128, 5, 192)])
def test_repack_paths(lanes_per_pool, packet_blocks, width, encoding):
    """Up to 64 packets and pools go to the kernel, more through the list:
    both sides of the line (64 or 128 packets, 64 or 128 pools), blocks of one
    to three lanes, a packet without blocks, a missing pool."""
    import torch
    from hw_b200 import filters as Fl
    import test_repack as R
    num_zmw, F = 128 * 64, 64
    table, data = R.make_chunk(num_zmw, 0, F, 64, packet_blocks, width, encoding)
    none = table[:1].copy()
    none["num_blocks"] = 0
    table = np.concatenate([table[:1], none, table[1:]])
    rp = Fl.Repacker(num_zmw, lanes_per_pool, F, "int16" if encoding == 0 else "uint8")
    chunks = rp.new_chunks()
    d = torch.from_numpy(data.copy()).cuda()
    rp(table, d, 0, chunks)
    want = R.oracle_repack(num_zmw, lanes_per_pool, F, encoding, table, data, 0)
    for got, w in zip(chunks, want):
        assert np.array_equal(got.cpu().numpy(), w)

    class Missing:
        def data_ptr(self):
            return 0
    with pytest.raises(HwError):
        rp(table, d, 0, chunks[:-1] + [Missing()])
