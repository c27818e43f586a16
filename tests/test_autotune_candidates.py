"""The autotuner's candidates: no two that launch the same kernel (no GPU needed)."""
import pytest

from gpufoam_b200 import autotune


@pytest.mark.parametrize("doubles", [500, 6000, 16000, 40000])
def test_candidates_differ(doubles):
    """To 128 unknowns the factorisation does not depend on lu_panel."""
    small, large = autotune.candidates(doubles, lu_panels=False), autotune.candidates(doubles)
    assert all(c["lu_panel"] == 0 for c in small) and all(c in large for c in small)
    keys = [tuple(sorted(c.items())) for c in large]
    assert len(set(keys)) == len(keys)
    fits = doubles * 8 <= 227 * 1024
    assert any(c["lu_panel"] == 4 for c in large) == fits
    assert sum(c["specialize"] for c in small) == (8 if fits else 4)


def test_tune_times_no_duplicates(monkeypatch):
    import torch
    timed = []

    class Solver:
        ode, mechs = None, [type("Mech", (), {"n_species": 53})()]

        def workspace_doubles(self):
            return 5600

        def set_launch(self, **cfg):
            self.cfg = cfg

    monkeypatch.setattr(autotune, "_key", lambda mechs, ode: "key")
    monkeypatch.setattr(autotune, "time_config", lambda s, cfg, *a, **k: timed.append(cfg) or float(len(timed)))
    as_tensor, full = torch.as_tensor, torch.full
    monkeypatch.setattr(torch, "as_tensor", lambda x, dtype=None, device=None: as_tensor(x, dtype=dtype))
    monkeypatch.setattr(torch, "full", lambda size, v, dtype=None, device=None: full(size, v, dtype=dtype))
    autotune.tune(Solver(), [[0.0]], 1e-6, use_cache=False)
    assert timed and all(c["lu_panel"] == 0 for c in timed)
