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


def _data(eng, slot, n):
    eng.seq_lens.data[slot] = n


def _dlpack(eng, slot, n):
    torch.from_dlpack(torch.utils.dlpack.to_dlpack(eng.seq_lens.view(-1)))[slot] = n


def _c_abi(eng, slot, n):
    eng._ck(eng._lib.vuib_set_seq_len(eng._handle, slot, n))


def _replayed_write(eng, slot, n):
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        eng.seq_lens[slot].fill_(n)
    eng.seq_lens[slot] = 3
    eng._rows[slot].rewind()   # the host's own write is the last that it sees
    g.replay()


def _c_step(eng, slot, n, call=None):
    """The backbone step of the C ABI on the engine's handle, `n` - 1 -> `n`."""
    import ctypes as C

    P = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    eng._rows[slot]._prompt_offset = n - 1
    eng._rows[slot].rewind()
    slots = torch.tensor([slot], dtype=torch.int32, device="cuda")
    codes = torch.zeros(1, eng.Q, dtype=torch.long, device="cuda")
    step = lambda: eng._ck(eng._lib.vuib_backbone_step(  # noqa: E731
        eng._handle, 1, P(slots), None, P(codes), P(eng._g_hidden_out), P(eng._g_cb0_out), P(eng._g_eos_out), eng._stream))
    if call is None:
        step()
    else:
        call(step)
    torch.cuda.synchronize()


def _replayed_step(eng, slot, n):
    def call(step):
        step()   # outside of a capture first: it loads the kernels
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            step()
        eng._rows[slot].rewind()
        g.replay()

    _c_step(eng, slot, n, call)


@pytest.mark.parametrize("write", [_data, _dlpack, _c_abi, _replayed_write, _c_step, _replayed_step])
def test_writers_that_the_host_does_not_see(nano_model, write):
    """Lengths written behind the Engine's back, just after it wrote them itself: the next prefill goes where the device says."""
    from vui_b200 import Engine

    eng = Engine(model=nano_model, max_rows=3, max_seq=128)
    rows = [eng.new_row() for _ in range(3)]
    ids = torch.randint(0, 1000, (9,), generator=torch.Generator().manual_seed(2))
    row, n = rows[1], 40
    eng.prefill_ids(row, ids)
    write(eng, row.idx, n)
    assert row.offset == n
    eng._kv.zero_()
    eng.prefill_ids(row, ids)
    assert row.offset == n + 9
    written = eng._kv[-1, 0, row.idx].flatten(1).any(dim=1).nonzero().flatten().tolist()
    assert written == list(range(n, n + 9))
    assert row.prefill([]) == n + 9 and row._prompt_offset == n + 9
    write(eng, row.idx, n)
    assert row.add_user("") == n
    eng.check_device()
