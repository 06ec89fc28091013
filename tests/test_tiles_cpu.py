"""Runs of tokens cut into tiles: the table that walking them one tile at a time gives."""

import numpy as np
import pytest
import torch

from bitexact_llm_b200.vllm_plugin import tri_prefill


@pytest.mark.parametrize("G,bm", [(4, 32), (1, 32), (8, 16), (32, 32), (5, 64), (64, 32)])
@pytest.mark.parametrize("lens", [[], [0], [1], [8, 0, 9], [31, 32, 33, 1, 1, 700]])
def test_tile_table(lens, G, bm):
    n = max(1, min(bm, 32) // G)
    pre, row = [], 0
    for i, q in enumerate(lens):
        pre.append((3 * i, row, q, q + 5))
        row += q
    want = [[r, t0 + s, min(n, q - s)] for r, t0, q, _ in pre for s in range(0, q, n)]
    got = tri_prefill.tile_table(pre, G, bm)
    assert got.dtype == torch.int32 and got.shape == (len(want), 3) and got.tolist() == want


@pytest.mark.parametrize("form", ["list", "lists", "iterator", "zip", "numpy", "tensor", "numpy rows", "tensor entries"])
def test_forms_of_the_runs(form):
    """Whatever can be walked row by row, and runs of no tokens or of fewer."""
    rows = [(4, 0, 20, 25), (1, 20, 0, 3), (0, 20, 9, 9), (2, 29, -3, 0), (7, 29, 1, 700)]
    pre = {"list": rows, "lists": [list(r) for r in rows], "iterator": iter(rows), "zip": zip(*zip(*rows)), "numpy": np.array(rows),
           "tensor": torch.tensor(rows), "numpy rows": [tuple(r) for r in np.array(rows)],
           "tensor entries": [tuple(r) for r in torch.tensor(rows)]}[form]
    want = [[r, t0 + s, min(8, q - s)] for r, t0, q, _ in rows for s in range(0, q, 8)]
    got = tri_prefill.tile_table(pre, 4)
    assert got.dtype == torch.int32 and got.tolist() == want
    with pytest.raises(ValueError):
        tri_prefill.tile_table([(4, 0, 20)], 4)
