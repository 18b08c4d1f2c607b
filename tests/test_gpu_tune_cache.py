"""The autotuner's cache file: an entry written for another variant table, or for
operators with other symmetry, is not taken."""
import pytest

from conftest import oracle  # noqa: F401

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import dgc_gb300 as dg  # noqa: E402
from dgc_gb300 import meshes  # noqa: E402


def test_entries_of_another_table_are_ignored(tmp_path, monkeypatch):
    cache = tmp_path / "tune.txt"
    monkeypatch.setenv("DGC_TUNE_CACHE", str(cache))
    D = dg.Discretization(meshes.jittered_square(6, 1), "maxwell_te", 5, dg.F32)

    def lines():
        return cache.read_text().split("\n")[:-1] if cache.exists() else []

    D.autotune(measure=False)  # empty cache: timed and stored
    key, chosen = lines()[0].split()
    parts = key.split("|")
    # the form of the key before it named the table, and other tables
    for other in ("|".join(parts[:6]), "|".join(parts[:-1] + ["table1"]), "|".join(parts[:-1] + ["table999"])):
        cache.write_text(f"{other} 0\n")
        D.autotune(measure=False)
        assert len(lines()) == 2 and lines()[1].split()[0] == key
    cache.write_text(f"{key} 0\n")  # its own entry is taken
    assert D.autotune(measure=False)[0] == 0 and len(lines()) == 1
    # operators without the reflection symmetry: variant 6 is another kernel
    Dr, Ds, L = (D.operator(w).copy() for w in (dg.OP_DR_WEAK, dg.OP_DS_WEAK, dg.OP_LIFT))
    Dr[1, 2] += 0.1
    D.set_operators(0, Dr, Ds, L)
    D.autotune(measure=False)
    assert len(lines()) == 2 and lines()[1].split()[0] != key
