"""The autotuner keeps no choice of the lines that get a warp which its sample
cannot tell (no GPU)."""

from __future__ import annotations

import numpy as np

from gpjson_b200 import tune


def test_no_warps_at_all_is_no_candidate():
    # with the cost lowest for -1, the search stays with the library's choice
    best, _ = tune.search(lambda s: 1.0 if s["long_line_bytes"] == -1 else 2.0)
    assert best["long_line_bytes"] == 0


def test_long_lines_searched_only_on_samples_with_some():
    short, long = np.arange(0, 800_000, 1600), np.array([0, 1600, 1600 + 8193])
    assert tune._candidates(short, 800_000)["long_line_bytes"] == [0]
    assert tune._candidates(np.array([0]), 8192)["long_line_bytes"] == [0]
    assert tune._candidates(np.array([0]), 8193) == tune.CANDIDATES
    assert tune._candidates(long, 9793 + 100) == tune.CANDIDATES


def test_stored_minus_one_is_left_to_the_library(tmp_path, monkeypatch):
    monkeypatch.setenv("GPJSON_TUNING_DIR", str(tmp_path))
    for var in tune.ENV.values():
        monkeypatch.delenv(var, raising=False)
    monkeypatch.setattr(tune, "_device_key_of", lambda device: "some_gpu")
    tune.save("some_gpu", {"index_ctas_per_sm": 3, "long_line_bytes": -1})
    set_to = []

    class Context:
        def set_tuning(self, **setting):
            set_to.append(setting)

    assert tune.apply(Context()) == {"index_ctas_per_sm": 3, "long_line_bytes": 0} == set_to[0]
    monkeypatch.setenv("GPJSON_LONG_LINE_BYTES", "-1")
    assert tune.apply(Context())["long_line_bytes"] == -1 == set_to[1]["long_line_bytes"]
    monkeypatch.delenv("GPJSON_LONG_LINE_BYTES")
    tune.save("some_gpu", {"long_line_bytes": 16384})
    assert tune.apply(Context()) == {"long_line_bytes": 16384}
