"""Rotary rows: two neighbouring frequencies a thread where the head size is a multiple of four, one otherwise; few
rows (the heads shared out over threads) and many."""

import pytest

from tests.test_gpu_prefill_bodies import test_rope_rows as check_rope_rows

pytestmark = [pytest.mark.gpu, pytest.mark.timeout(120)]


@pytest.mark.parametrize("rows,heads,kv_heads,dim", [
    (5, 3, 1, 66), (7, 2, 2, 2), (9, 5, 1, 4), (33, 3, 3, 68), (3000, 9, 1, 66), (6000, 4, 1, 128),
])
def test_head_sizes(rows, heads, kv_heads, dim):
    check_rope_rows(rows, heads, kv_heads, dim)
