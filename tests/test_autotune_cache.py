"""What the tuner's cache and its choice at 256^3 depend on (no GPU)."""
import json

import pytest

import smectic3d_b200 as S
from smectic3d_b200 import autotune


@pytest.fixture
def timed(monkeypatch, tmp_path):
    monkeypatch.setenv("SMECTIC_B200_CACHE", str(tmp_path / "tuned.json"))
    monkeypatch.setattr(autotune, "_gpu_name", lambda: "FakeGPU")
    calls = []

    def use(us):
        monkeypatch.setattr(autotune, "_time_variant", lambda p, v, steps: (calls.append(v), us[v] * 1e-6)[1])
        return calls
    return tmp_path / "tuned.json", use


def test_an_entry_timed_with_other_kernels_is_timed_again(timed):
    """Entries without a digest of the kernels (the former format) and with another one."""
    cache, use = timed
    p = S.Params(n=128, precision="fp32")
    old = {"variant": 2, "us_per_step": {"1": 30.0, "2": 20.0}, "replica_block": 0, "pencil_tile": 0}
    for entry in (old, {**old, "kernels": "other"}):
        cache.write_text(json.dumps({autotune._key(p, "FakeGPU"): entry}))
        calls = use({1: 15.0, 2: 25.0, 4: 35.0})
        assert autotune.tune(p, steps=3)["variant"] == 1 and calls
        del calls[:]
        assert autotune.tune(p, steps=3)["variant"] == 1 and not calls


@pytest.mark.parametrize("prec,default", [("fp32", 8), ("fp32_u64", 8), ("fp64", 16)])
def test_noise_does_not_move_the_cluster_size_of_256(timed, prec, default):
    _, use = timed
    p = S.Params(n=256, precision=prec)
    use({4: 131.0, 8: 132.0, 16: 132.5})
    assert autotune.tune(p, steps=3, use_cache=False)["variant"] == default
    use({4: 110.0, 8: 132.0, 16: 132.5})
    assert autotune.tune(p, steps=3, use_cache=False)["variant"] == 4
