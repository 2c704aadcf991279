"""FP64 candidates of the autotuner: the one-thread kernels' four, and several
threads per system where a system has rows for them; results cached for other
kernels are not applied."""
import json


def test_candidates():
    from ntk import autotune

    one = [{"f64_x_variant": v, "f64_threads": t} for v in (0, 1) for t in (64, 128)]
    assert autotune.candidates("fp64", 16) == one
    assert autotune.candidates("fp64", 512) == one + [{"f64_chunks": 2}]
    assert {"f64_chunks": 2} not in autotune.candidates("fp32_refine", 512)


class FakePlan:
    n, precision = 700, "fp32_refine"

    def __init__(self):
        self.cfg = {}

    def set_tuning(self, **kw):
        self.cfg.update(kw)


def test_results_of_other_kernels_are_not_applied(tmp_path, monkeypatch):
    """A cache of before the kernel set was part of the key, and one of
    another kernel set: both could hold a value that now means another kernel."""
    from ntk import autotune

    monkeypatch.setenv("NTK_AUTOTUNE_CACHE", str(tmp_path / "cache.json"))
    monkeypatch.setattr(autotune, "device_name", lambda: "FAKE-GPU")
    old = {"config": {"refine_kernel": 1, "refine_w": 4}, "ms": 1.0, "all": []}
    keys = ["FAKE-GPU|700|fp32_refine|x"]
    with monkeypatch.context() as m:
        m.setattr(autotune, "KERNEL_SET", autotune.KERNEL_SET + 1)
        keys.append(autotune.cache_key(FakePlan(), "x"))
    (tmp_path / "cache.json").write_text(json.dumps({k: old for k in keys}))
    p = FakePlan()
    assert autotune.apply_cached(p, "x") is None and p.cfg == {}
    timed = []
    res = autotune.tune(p, lambda: None, "x", timer=lambda run, repeats: timed.append(1) or float(len(timed)))
    assert timed and res["config"] == autotune.candidates("fp32_refine", 700)[0]
    q = FakePlan()
    assert autotune.apply_cached(q, "x") == res["config"] and q.cfg == res["config"]
