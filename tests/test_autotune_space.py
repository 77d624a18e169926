"""The autotuner times no launch shape twice for the same figure: sweep_warps 1
is taken as 2 (two warps sweep a pass), so the space holds one of them."""
from skity_gb300 import autotune


class _Batch:
    def __init__(self):
        self.cfg, self.timed = None, []

    def set_config(self, **cfg):
        self.cfg = cfg

    def render(self):
        shape = dict(self.cfg, sweep_warps=max(2, self.cfg["sweep_warps"]))
        self.timed.append(tuple(sorted(shape.items())))
        return {"composite_ms": 1.0, "device_ms": 1.0}


def test_no_launch_shape_is_timed_twice(tmp_path, monkeypatch):
    monkeypatch.setenv("SKITY_GB300_TUNE_CACHE", str(tmp_path / "tune.json"))
    b = _Batch()
    r = autotune.tune(b, "k", reps=1, use_cache=False)
    launch = lambda t: tuple(sorted(dict(t, sweep_warps=max(2, t["sweep_warps"])).items()))  # noqa: E731
    for key in ("composite_ms", "device_ms"):
        shapes = [launch({k: v for k, v in t.items() if not k.endswith("_ms")})
                  for t in r["trials"] if key in t]
        assert shapes and len(set(shapes)) == len(shapes), key
