"""Row.offset and the position a prefill starts at, whoever wrote the lengths last: the host (reset, rewind, prefill), generated frames
and replays of a captured one, or a caller writing seq_lens through any of its views, inside inference mode and out of it."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [True, False])
@pytest.mark.parametrize("rows", [1, 5])
def test_lengths_are_what_the_device_has(nano_model, rows, mode):
    from vui_b200 import Engine

    with torch.inference_mode(mode):
        eng = Engine(model=nano_model, max_rows=rows, max_seq=256)
        rs = [eng.new_row() for _ in range(rows)]
    ids = torch.randint(0, 1000, (9,), generator=torch.Generator().manual_seed(1))

    def check(want):
        assert [r.offset for r in rs] == want == eng.seq_lens[:rows].tolist()

    with torch.inference_mode(mode):
        check([0] * rows)
        h = torch.stack([eng.prefill_ids(r, ids) for r in rs])
        check([9] * rows)
        eng.prefill_ids(rs[0], ids)
        check([18] + [9] * (rows - 1))
        rs[0]._prompt_offset = 4
        rs[0].rewind()
        check([4] + [9] * (rows - 1))
        eng.generate_frames(rs, h, 4, greedy=True)
        moved = eng.seq_lens[:rows].tolist()
        assert moved[0] > 4
        check(moved)
        rs[0].reset()
        g = eng._frame_graph(rows)
        eng._g_slot_idx[:rows] = torch.arange(rows, dtype=torch.int32, device="cuda")
        eng._g_seq_inc[:rows] = 1
        rs[0].reset()
        g.replay()
        check([1] + [n + 1 for n in moved[1:]])
        rs[-1].reset()
        eng.flash_kv_caches[3].seq_lens[rows - 1] = 7
        check(([1] + [n + 1 for n in moved[1:]])[:-1] + [7])
        rs[-1].reset()
        eng.seq_lens.fill_(20)
        eng.prefill_ids(rs[-1], ids)
        check([20] * (rows - 1) + [29])
        rs[-1].rewind()
        eng.seq_lens.copy_(torch.full((rows + 1,), 250, dtype=torch.int32))
        with pytest.raises(RuntimeError, match="overflows"):
            eng.prefill_ids(rs[-1], ids)
    eng.check_device()
