"""FP64 candidates of the autotuner: the one-thread kernels' four, and several
threads per system where a system has rows for them."""


def test_candidates():
    from ntk import autotune

    one = [{"f64_x_variant": v, "f64_threads": t} for v in (0, 1) for t in (64, 128)]
    assert autotune.candidates("fp64", 16) == one
    assert autotune.candidates("fp64", 512) == one + [{"f64_chunks": 2}]
    assert {"f64_chunks": 2} not in autotune.candidates("fp32_refine", 512)
