"""The autotuner's choice among timed launches, without a GPU: the library's
own choice is a candidate, is kept unless another is more than 1% faster, and
a cache entry made without it is not used."""

import json
from types import SimpleNamespace

import pytest

from SWESimulators import Autotune, _native


def test_the_librarys_choice_is_a_candidate():
    assert Autotune.DOMAIN_CANDIDATES[0] == (_native.GO_SHAPE_AUTO, 0)
    assert Autotune.BATCH_CANDIDATES[0] == (_native.GO_SHAPE_AUTO, 0, 0)


def _simulator(land=False, default_us=16.6, other_us=28.8):
    sim = SimpleNamespace(nx=512, ny=512, r=0.0, linear_friction=False, dt=1.0, gpu_stream=None, launch=None,
                          wind_stress=SimpleNamespace(is_uniform=lambda: True))

    def set_launch(shape, rows):
        sim.launch = (shape, rows)
    sim._domain = SimpleNamespace(set_launch=set_launch, may_have_land=land, bc=(1, 1, 1, 1))
    sim._launch_steps = lambda n, dt, w: None
    sim.time = lambda: default_us if sim.launch[0] == _native.GO_SHAPE_AUTO else other_us + sim.launch[1] * 1e-3
    return sim


@pytest.fixture
def timed(monkeypatch, tmp_path):
    monkeypatch.setenv("GOCEAN_TUNE_CACHE", str(tmp_path / "tune.json"))
    monkeypatch.setattr(Autotune, "_device_name", lambda: "B200")
    monkeypatch.setattr(Autotune, "_snapshot", lambda sims: None)
    monkeypatch.setattr(Autotune, "_restore", lambda sims, snap: None)
    monkeypatch.setattr(_native, "require_cuda", lambda: SimpleNamespace(cuda=SimpleNamespace(synchronize=lambda: None)))
    current = {}
    monkeypatch.setattr(Autotune, "_time", lambda fn, stream, repeats=3: current["sim"].time())

    def tune(sim):
        current["sim"] = sim
        return Autotune.tune_domain(sim)
    return tune


@pytest.mark.parametrize("default_us,other_us,kept", [(16.6, 28.8, True), (28.8, 28.8, True), (29.0, 28.8, True),
                                                      (29.2, 28.8, False)])
def test_default_is_kept_unless_another_is_faster(timed, default_us, other_us, kept):
    sim = _simulator(default_us=default_us, other_us=other_us)
    best, info = timed(sim)
    assert (best == (_native.GO_SHAPE_AUTO, 0)) == kept and sim.launch == best
    again, hit = timed(sim)
    assert again == best and sim.launch == best


def test_cache_entries_without_the_default_are_not_used(timed):
    with open(Autotune.cache_path(), "w") as fh:
        json.dump({"domain|B200|512x512|r0-lf0-ws0": {"launch": [4, 8]}}, fh)
    assert timed(_simulator())[0] == (_native.GO_SHAPE_AUTO, 0)
    # nor is the entry of a domain without land for one with it
    best, _ = timed(_simulator(land=True, default_us=40.0))
    assert best != (_native.GO_SHAPE_AUTO, 0)
