"""Prompts longer than one prefill call: cut at the limit that was asked for, or at the default's 1024 rows, with the same result bit for
bit as in other pieces."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("limit,n", [(256, 256), (256, 300), (512, 513), (None, 1024), (None, 1500), (None, 2000)])
def test_a_long_prompt_is_cut_at_the_limit(nano_model, limit, n):
    from vui_b200 import Engine

    eng = Engine(model=nano_model, max_rows=2, max_seq=2048, **({} if limit is None else {"max_prefill_rows": limit}))
    ids = torch.randint(0, 151936, (n,), generator=torch.Generator().manual_seed(n))
    r1, r2 = eng.new_row(), eng.new_row()
    rows = 1024 if limit is None else limit
    before = eng.launch_count()
    eng.prefill_ids(r1, ids[:1])
    call = eng.launch_count() - before   # a call's launches do not depend on its rows
    eng._rewind_row(r1, 0)
    h1 = eng.prefill_ids(r1, ids)
    assert eng.launch_count() - before == call * (1 + -(-n // rows))
    for t in range(0, n, 100):
        h2 = eng.prefill_ids(r2, ids[t:t + 100])
    eng.check_device()
    assert r1.offset == r2.offset == n and torch.equal(h1, h2)
    assert torch.equal(eng._kv[:, :, r1.idx, :n], eng._kv[:, :, r2.idx, :n])
