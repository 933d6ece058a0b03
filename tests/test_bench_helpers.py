"""bench.py's host-side helpers (CPU only): the reference's command line of a
job spec, and the reference legs' absence where the reference was not built."""
from __future__ import annotations

import importlib.util
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent


def _bench():
    spec = importlib.util.spec_from_file_location("bench_mod", ROOT / "bench.py")
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    return mod


def test_spec_args_are_the_reference_options():
    b = _bench()
    args = b._spec_args(dict(pmin=42 * 10**12, pmax=42 * 10**12 + 10**6, kmin=1201, kmax=9999, nmin=2000000,
                             nmax=3000000))
    assert args == ["-p42000000000000", "-P42000001000000", "-k1201", "-K9999", "-n2000000", "-N3000000"]
    riesel = b._spec_args(dict(pmin=10**12, pmax=10**12 + 10, kmin=3, kmax=5, nmin=100, nmax=200, sign=-1))
    assert riesel[-1] == "-R"


def test_reference_legs_absent_without_a_build(tmp_path):
    b = _bench()
    b.REF_CUDA_BIN = tmp_path / "missing"
    b.REF_CUDA_TWIN_BIN = tmp_path / "missing_twin"
    assert b.reference_gpu_sample(None) is None
    assert b.reference_gpu_sample(None, twin=True) is None
    assert b.reference_gpu_sample(None, binary=tmp_path / "missing_dropin") is None
    b.REF_BIN = tmp_path / "missing_cpu"
    assert b.reference_sample(1.0) is None


def test_tensor_roofline_is_work_over_a_measured_peak(monkeypatch):
    """The fraction is the matrix products' (fixed by the method) and does not move
    with the kernel's own instruction count, which only says how busy it is."""
    b = _bench()
    rows = []
    for instr in (4000.0, 2000.0):
        monkeypatch.setattr(b, "_from_profile", lambda _, key, i=instr: {"mma_flop_per_prime": 3.0e6}.get(key, i))
        rows.append(b._tensor_roofline("k_tensor_walk", 2.0e8, 2000.0, 100, 1500.0))
    assert rows[0]["bound"] == "tensor" and abs(rows[0]["frac"] - 0.4) < 1e-12
    assert rows[0]["frac"] == rows[1]["frac"]
    assert abs(rows[0]["issue_slots"]["busy"] - 1.0) < 1e-12 and abs(rows[1]["issue_slots"]["busy"] - 0.5) < 1e-12
