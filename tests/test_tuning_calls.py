"""What the tuner's answer is used for (no GPU: the device calls are stand-ins)."""
import numpy as np
import torch

from hindemith_b200 import _lib as L
from hindemith_b200 import autotune, device, frontend, hs_average_stencil


def run_hs_loop(monkeypatch, defines, answers):
    """The hs_config of a fused loop under `defines`; answers[passes_only]: the tuner's answer."""
    seen = []
    monkeypatch.setattr(autotune, "best_sweep_config",
                        lambda H, W, ld, fast_math, passes_only=False: answers[passes_only])
    monkeypatch.setattr(device, "_same_layout", lambda *ts: ts)
    monkeypatch.setattr(device, "hs_sweeps", lambda *a: seen.append(a[-1]))
    plane = torch.zeros(8, 12)
    env = dict(Ix=plane, Iy=plane, It=plane, u=plane, v=plane, alpha2=np.float32(1), A=hs_average_stencil())
    ex = frontend.Executor(frontend.parse("def f(u):\n    return u\n", {"u": frontend.ARRAY2D}), defines)
    info = dict(A="A", Ix="Ix", Iy="Iy", It="It", U="u", V="v", alpha2="alpha2")
    ex._hs_sweeps(frontend.Stmt("HSSweeps", info=info, ub=5), env)
    return seen[0]


def test_a_given_segment_is_combined_with_a_tuned_depth(monkeypatch):
    """The library's own choice (0, 0, 0) is none to combine with the user's rows: with them it
    would be the passes at the default depth, which nobody timed."""
    answers = {False: (0, 0, 0), True: (5, 24, 2)}
    cfg = run_hs_loop(monkeypatch, {"hs_rows_per_segment": 40, "hs_fast_math": True}, answers)
    assert (cfg.sweeps_per_pass, cfg.rows_per_segment, cfg.layout) == (5, 40, 2)
    cfg = run_hs_loop(monkeypatch, {"hs_fast_math": True}, answers)
    assert (cfg.sweeps_per_pass, cfg.rows_per_segment, cfg.layout) == (0, 0, 0)


def test_a_tuning_among_the_passes_is_cached_apart():
    a = autotune._sweep_key("B200", 480, 640, 640, True, autotune.DEFAULT_TUNING_SWEEPS)
    b = autotune._sweep_key("B200", 480, 640, 640, True, autotune.DEFAULT_TUNING_SWEEPS, True)
    c = autotune._sweep_key("B200", 480, 640, 640, True, 77, True)
    assert len({a, b, c}) == 3


def test_a_cache_file_keeps_apart_what_answers_were_chosen_from(monkeypatch, tmp_path):
    """Answers from before the library's own choice was timed are not taken for this tuner's, and
    stay in the file; its own are read back."""
    import json

    path = tmp_path / "cache.json"
    key = autotune._sweep_key("B200", 1080, 1920, 1920, True, 500)
    path.write_text(json.dumps({key: [7, 0, 2]}))
    monkeypatch.setenv("HS_AUTOTUNE_CACHE", str(path))
    monkeypatch.setattr(autotune, "_cache", {})
    autotune._load_file()
    assert key not in autotune._cache
    autotune._cache[key] = (0, 0, 0)
    autotune._save_file()
    monkeypatch.setattr(autotune, "_cache", {})
    autotune._load_file()
    assert autotune._cache == {key: (0, 0, 0)}
    assert json.loads(path.read_text())[key] == [7, 0, 2]
    path.write_text("not json")
    autotune._load_file()
    autotune._save_file()
    assert list(json.loads(path.read_text()).values()) == [[0, 0, 0]]


def test_every_candidate_is_warmed_up(monkeypatch):
    """The call before the timed ones launches the candidate's kernel: at depth 0 too."""
    class Event:
        def __init__(self, enable_timing):
            pass

        def record(self):
            pass

        def synchronize(self):
            pass

        def elapsed_time(self, other):
            return 1.0

    calls = []
    monkeypatch.setattr(torch.cuda, "Event", Event)
    monkeypatch.setattr(device, "hs_sweeps", lambda *a: calls.append((a[4], a[-1].sweeps_per_pass)))
    for T in (0, 1, 4, 7):
        calls.clear()
        autotune.time_config(*[None] * 5, T, 0, True, 240, reps=2)
        assert calls == [(max(T, 2), T), (240, T), (240, T)]
