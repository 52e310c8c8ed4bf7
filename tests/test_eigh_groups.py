"""
Host logic around side-by-side eigendecompositions and scratch memory: matrices and solver workspaces held at once are
bounded, and where there is no memory for that, calls go on with less.
"""
from __future__ import annotations

import pytest
import torch

from fasterlmm_gb300 import core

OOM = torch.cuda.OutOfMemoryError


@pytest.mark.parametrize("sizes", [[], [5], [3000] * 30, [20_000, 100, 20_000, 100, 100], [8000] * 3 + [100] * 40])
def test_groups_cover_and_stay_within_the_bound(sizes):
    groups = core.eigh_groups(sizes)
    assert [i for g in groups for i in g] == list(range(len(sizes)))
    for g in groups:
        held = sum(8 * sizes[i] ** 2 for i in g)
        work = min(len(g), core.EIGH_WORKERS) * 16 * max(sizes[i] for i in g) ** 2
        assert len(g) == 1 or held + work <= core.EIGH_MANY_BYTES


def _run(monkeypatch, most: int, sizes):
    """eigh_each with memory for `most` matrices at a time; what was decomposed together."""
    together = []

    def many(mats):
        if len(mats) > most:
            raise OOM("out of memory")
        together.append(len(mats))
        return [m.diagonal().clone() for m in mats]

    monkeypatch.setattr(core, "eigh_many", many)
    out = list(core.eigh_each(sizes, lambda i: torch.full((sizes[i], sizes[i]), float(i))))
    assert [i for i, _, _ in out] == list(range(len(sizes)))
    for i, evals, V in out:
        assert evals.tolist() == [float(i)] * sizes[i] and V.shape == (sizes[i], sizes[i])
    return together


def test_matrices_go_together_or_one_by_one(monkeypatch):
    assert _run(monkeypatch, 10, [2, 3, 4, 5]) == [4]
    assert _run(monkeypatch, 3, [2, 3, 4, 5]) == [1, 1, 1, 1]
    monkeypatch.setattr(core, "EIGH_MANY_BYTES", 8 * 25 * 2 + 16 * 25 * 2)
    assert _run(monkeypatch, 1, [5, 5, 5]) == [1, 1, 1]
    assert _run(monkeypatch, 2, [5, 5, 5]) == [2, 1]
    with pytest.raises(OOM):
        _run(monkeypatch, 0, [2, 3])


def test_scratch_that_does_not_fit_is_asked_for_in_halves(monkeypatch):
    w = core._Work()
    asked = []

    def get(dev, nbytes):
        asked.append(nbytes)
        if nbytes > 5 << 20:
            raise OOM("out of memory")
        return None, nbytes

    monkeypatch.setattr(w, "get", get)
    assert w.up_to(torch.device("cpu"), 40 << 20) == (None, 5 << 20)
    assert asked == [40 << 20, 20 << 20, 10 << 20, 5 << 20]
    monkeypatch.setattr(w, "get", lambda dev, nbytes: (_ for _ in ()).throw(OOM("out of memory")))
    with pytest.raises(OOM):
        w.up_to(torch.device("cpu"), 40 << 20)
