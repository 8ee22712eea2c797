"""The autotuner's grids hold the library's default settings, and it keeps the default sort unless
another one is faster by more than noise (timings replaced by a table; nothing is launched)."""
import inspect

import pytest


@pytest.fixture()
def tuner(wf, monkeypatch):
    from vulkanwavefrontpathtracer_gb300 import autotune

    def use(ms):
        """ms(knob reader) -> the time of one measurement"""
        monkeypatch.setattr(autotune, "_timeit", lambda fn, *a, **k: ms(wf.api.tune_get))
        return autotune
    return use


def test_traversal_grid_holds_the_defaults(wf, tuner):
    p = inspect.signature(tuner(lambda get: 1.0).tune_traversal).parameters
    get = wf.api.tune_get
    for name, knobs in (("refills", ["refill"]), ("postpones", ["postpone"]), ("coops", ["coop"]),
                        ("batches", ["batch", "any_batch"]), ("steps", ["steps", "any_steps"])):
        for k in knobs:
            assert get("trace.bvh8." + k) in p[name].default, (name, k)


@pytest.mark.parametrize("bits,dtype", [(32, "int32"), (63, "int64")])
@pytest.mark.parametrize("other,gain,kept", [(2, 0.0, True), (2, 0.01, True), (2, 0.1, False), (1, 0.5, False)])
def test_sort_keeps_the_default(wf, tuner, bits, dtype, other, gain, kept):
    import torch
    calls = []

    def ms(get):
        calls.append(1)
        if len(calls) % 2:
            return 0.5  # the keys' copy
        return 1.5 - (gain if (get("sort.digit_bits"), get("sort.tiles")) == (8, other) else 0.0)

    got = tuner(ms).tune_sort(torch.zeros(1000, dtype=getattr(torch, dtype)), bits)
    assert (got["digit_bits"], got["tiles"]) == ((8, 0) if kept else (8, other))
    assert {(e["digit_bits"], e["tiles"]) for e in got["table"]} >= {(8, t) for t in (0, 1, 2)}
    assert wf.api.tune_get("sort.tiles") == 0 and wf.api.tune_get("sort.digit_bits") == 8
