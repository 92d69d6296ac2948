"""Autotuner logic on a scripted engine (no GPU): candidate timing,
refused candidates, selection, cache round trip, batch-width choice."""

from __future__ import annotations

import numpy as np
import pytest

from magnelio_b200 import autotune
from magnelio_b200._lib import FitbError


class ScriptedEngine:
    """Stands in for FitEngine: time_stencil returns a per-configuration
    time; some configurations are refused like the C ABI refuses them."""

    def __init__(self, times, refuse=()):
        self.times = times
        self.refuse = set(refuse)
        self.cfg = None
        self.log = []

    def configure_stencil(self, kind, variant=0, ichunk=0):
        if (kind, variant, ichunk) in self.refuse:
            raise FitbError(-1, "refused")
        self.cfg = (kind, variant, ichunk)
        self.log.append(self.cfg)

    def time_stencil(self, n):
        t = self.times[self.cfg]
        return t * 0.5, t * 0.5

    def close(self):
        pass


def test_tune_engine_picks_the_fastest_and_skips_refused():
    cands = [("stream", 0, 0), ("stream", 0, 32), ("vec", 3, 0), ("bulk", 0, 0)]
    times = {("stream", 0, 0): 1.0, ("stream", 0, 32): 0.8, ("vec", 3, 0): 1.5, ("bulk", 0, 0): 0.1}
    eng = ScriptedEngine(times, refuse={("bulk", 0, 0)})
    best, table = autotune.tune_engine(eng, cands, iters=3)
    assert best[:3] == ("stream", 0, 32) and best[3] == pytest.approx(0.8)
    assert len(table) == 3
    assert eng.cfg == ("stream", 0, 32)  # left configured with the winner


def test_tune_engine_with_nothing_runnable_is_an_error():
    eng = ScriptedEngine({}, refuse={("stream", 0, 0)})
    with pytest.raises(RuntimeError, match="no stencil candidate"):
        autotune.tune_engine(eng, [("stream", 0, 0)])


class _Prob:
    nx, ny, nz, dt = 10, 12, 14, 1e-12
    cpml = []


def test_tune_problem_caches_and_picks_the_best_batch(tmp_path, monkeypatch):
    monkeypatch.setenv("FITB_TUNE_CACHE", str(tmp_path / "tune.json"))
    built = []

    def fake_scratch(prob, B, precision, device, coef):
        built.append(B)
        # per-pass time grows slower than B: B = 4 has the best throughput
        base = {1: 1.0, 2: 1.6, 4: 2.4, 8: 6.0}[B]
        return ScriptedEngine({("stream", 0, 0): base, ("stream", 0, 16): base * 0.9})

    monkeypatch.setattr(autotune, "_scratch_engine", fake_scratch)
    cands = [("stream", 0, 0), ("stream", 0, 16)]
    res = autotune.tune_problem(_Prob(), batch_widths=(1, 2, 4, 8), candidates=cands)
    assert res.batch == 4 and res.config() == ("stream", 0, 16)
    assert res.ms == pytest.approx(2.16)
    assert sorted(built) == [1, 2, 4, 8]
    # second call: every width comes from the cache
    built.clear()
    again = autotune.tune_problem(_Prob(), batch_widths=(1, 2, 4, 8), candidates=cands)
    assert built == [] and again.config() == res.config() and again.batch == 4
    # the cache is plain JSON with one entry per width
    import json

    data = json.loads((tmp_path / "tune.json").read_text())
    assert len(data) == 4 and all("|B" in k for k in data)


def test_apply_configures_the_engine():
    eng = ScriptedEngine({("vec", 2, 24): 1.0})
    autotune.apply(eng, autotune.TuneResult("vec", 2, 24, 1, 1.0, 1.0))
    assert eng.cfg == ("vec", 2, 24)
    assert np.isfinite(1.0)


def test_cache_keys_name_the_candidate_set():
    """A result tuned over another candidate set is not reused: the key
    carries the set's version."""
    k = autotune.cache_key(64, 64, 64, 1, "single", "native", 6, "B200")
    assert k.endswith(f"|c{autotune.CANDIDATE_SET}")
    assert ("fused", 7, 0) in autotune.DEFAULT_CANDIDATES  # the tile form is tuned


class SlabEngine(ScriptedEngine):
    """A slab step without a depth runs on the direct kernels; 16-bit storage
    refuses "simple"."""

    def stencil_config(self):
        kind, variant, ichunk = self.cfg or ("simple", 0, 0)
        return {"kind": kind, "variant": variant, "ichunk": ichunk}

    def time_stencil(self, n):
        self.timed = [*getattr(self, "timed", []), self.cfg]
        return super().time_stencil(n)


def test_the_same_kernels_are_timed_once():
    cands = [("simple", 0, 0), ("fused", 16, 0), ("fused", 17, 0), ("fused", 16, 16)]
    times = {("simple", 0, 0): 1.0, ("fused", 16, 0): 0.99, ("fused", 17, 0): 0.98, ("fused", 16, 16): 2.0}
    eng = SlabEngine(times)
    best, table = autotune.tune_engine(eng, cands)
    assert [r[:3] for r in table] == [("simple", 0, 0), ("fused", 16, 16)] and best[0] == "simple"
    # where "simple" is refused, the first slab step stands for them
    eng = SlabEngine(times, refuse={("simple", 0, 0)})
    best, table = autotune.tune_engine(eng, cands)
    assert [r[:3] for r in table] == [("fused", 16, 0), ("fused", 16, 16)] and best[:2] == ("fused", 16)


def test_the_slab_step_is_tuned_on_its_unit_lists_too():
    slabs = [c for c in autotune.DEFAULT_CANDIDATES if c[0] == "fused" and c[1] >= autotune.SLAB_VARIANT_BASE]
    for depth in (0, 16):
        assert {c[1] for c in slabs if c[2] == depth} == set(range(16, 26))
    # without dead units every form of depth 0 is the direct kernels: one of them is timed
    times = {c: 1.0 for c in autotune.DEFAULT_CANDIDATES}
    _, table = autotune.tune_engine(SlabEngine(times), autotune.DEFAULT_CANDIDATES)
    assert not [r for r in table if r[0] == "fused" and r[1] >= autotune.SLAB_VARIANT_BASE and r[2] == 0]
    assert len({r[:3] for r in table}) == len(table)


def test_sixteen_bit_coefficients_are_tuned_against_the_handle_as_it_comes(tmp_path, monkeypatch):
    monkeypatch.setenv("FITB_TUNE_CACHE", str(tmp_path / "tune.json"))
    eng = SlabEngine({None: 0.5, ("stream", 0, 0): 1.0, ("vec", 3, 0): 2.0}, refuse={("simple", 0, 0)})
    monkeypatch.setattr(autotune, "_scratch_engine", lambda *a: eng)
    cands = [("simple", 0, 0), ("stream", 0, 0), ("vec", 3, 0)]
    res = autotune.tune_problem(_Prob(), coef="bf16", candidates=cands)
    assert res.config() == ("default", 0, 0) and len(res.table) == 3
    fresh = ScriptedEngine({})
    autotune.apply(fresh, res)
    assert fresh.log == []
    native = autotune.tune_problem(_Prob(), candidates=cands, use_cache=False)
    assert native.kind == "stream"
