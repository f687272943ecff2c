"""Kernels of a step at the edges of their ranges: first and last sizes of a tile or a dispatch rule, remainders, odd sizes."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from vox_serve_b200 import ops as o

    return o


def _i32(v):
    return torch.tensor(v, dtype=torch.int32, device="cuda")


@pytest.mark.parametrize("new,old,pad", [
    ([1], [0], 0), ([3, 0, 5, 0, 0, 2], [0, 4, 15, 0, 16, 33], 7), ([0, 0, 9], [3, 0, 0], 0), ([1024], [5], 0), ([1025, 1], [0, 0], 3),
    ([1] * 1023 + [0], [7] * 1024, 1), ([2, 1] * 600, [1, 40] * 600, 24),      # request tables on both sides of the one in shared memory
])
def test_plan_rows_prefill(ops, new, old, pad):
    page, chunk, n = 16, 16, len(new)
    kv = [max(a + b, 1) for a, b in zip(new, old)]
    pages = [(x + page - 1) // page for x in kv]
    qo, ip = np.concatenate([[0], np.cumsum(new)]).tolist(), np.concatenate([[0], np.cumsum(pages)]).tolist()
    idx = np.random.RandomState(n).permutation(ip[-1]).tolist()
    T = qo[-1]
    plan = ops.RowPlan(T + pad, "cuda")
    ops.plan_rows(plan, _i32(qo), _i32(ip), _i32(idx), _i32([(x - 1) % page + 1 for x in kv]), n, T + pad, page, chunk)
    req, at = [], []
    for r in range(n):
        req += [r] * new[r]
        at += [kv[r] - new[r] + j for j in range(new[r])]
    assert plan.row_req[:T + pad].tolist() == req + [-1] * pad
    assert plan.row_kvlen[:T + pad].tolist() == [g + 1 for g in at] + [0] * pad
    assert plan.row_page[:T + pad].tolist() == [idx[ip[r] + g // page] for r, g in zip(req, at)] + [-1] * pad
    assert plan.row_slot[:T].tolist() == [g % page for g in at]
    assert plan.row_pagebase[:T].tolist() == [ip[r] for r in req] and plan.row_old[:T].tolist() == [kv[r] - new[r] for r in req]
    chunks = [(g + chunk) // chunk for g in at] + [0] * pad
    assert plan.row_chunk_start[:T + pad + 1].tolist() == [0] + np.cumsum(chunks).tolist()
