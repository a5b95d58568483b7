"""The step's scratch allocator (qwen_engine_b200/parts/base.py: Arena) on the CPU: stack discipline for
the layers' intermediates, memory that lives for the whole step beside it, growth after an overflow."""
import torch

from qwen_engine_b200.parts.base import Arena


def _span(t):
    return t.data_ptr(), t.data_ptr() + t.numel() * t.element_size()


def _overlap(a, b):
    (a0, a1), (b0, b1) = _span(a), _span(b)
    return a0 < b1 and b0 < a1


def test_layers_reuse_their_scratch_and_step_memory_survives_them():
    ar = Arena("cpu", 1 << 16)
    ar.reset()
    m = ar.mark()
    a = ar.alloc((10, 64), torch.float32)
    table = ar.alloc_step((8, 64, 2), torch.float32)           # made inside the first layer's frame
    b = ar.alloc((10, 64), torch.float32)
    ar.release(m)
    for _ in range(3):                                         # the next layers: the same frame again
        m = ar.mark()
        a2 = ar.alloc((10, 64), torch.float32)
        c = ar.alloc((40, 64), torch.float32)                  # more than the first layer took after `a`
        assert a2.data_ptr() == a.data_ptr()
        assert not _overlap(c, table) and not _overlap(a2, table)
        ar.release(m)
    assert not _overlap(b, table)
    # the same sequence in the next step gives the same addresses (steps replayed from CUDA graphs rely on it)
    ar.reset()
    m = ar.mark()
    assert ar.alloc((10, 64), torch.float32).data_ptr() == a.data_ptr()
    assert ar.alloc_step((8, 64, 2), torch.float32).data_ptr() == table.data_ptr()


def test_bump_and_step_allocations_never_meet():
    ar = Arena("cpu", 4096)
    ar.reset()
    s1 = ar.alloc_step((256,), torch.float32)                  # 1 KB from the far end
    x = ar.alloc((512,), torch.float32)                        # 2 KB from the near end
    y = ar.alloc((512,), torch.float32)                        # does not fit between them: a tensor of its own
    s2 = ar.alloc_step((512,), torch.float32)                  # nor does this
    ts = [s1, x, y, s2]
    assert all(not _overlap(p, q) for i, p in enumerate(ts) for q in ts[i + 1:])
    assert ar._overflow
    ar.reset()                                                 # grown: now everything fits in the buffer
    lo, hi = ar.buffer.data_ptr(), ar.buffer.data_ptr() + ar.capacity
    ts = [ar.alloc_step((256,), torch.float32), ar.alloc((512,), torch.float32), ar.alloc((512,), torch.float32),
          ar.alloc_step((512,), torch.float32)]
    assert not ar._overflow
    assert all(lo <= _span(t)[0] and _span(t)[1] <= hi for t in ts)
    assert all(not _overlap(p, q) for i, p in enumerate(ts) for q in ts[i + 1:])


def test_a_remembered_view_is_not_handed_out_over_step_memory():
    ar = Arena("cpu", 4096)
    ar.reset()
    big = ar.alloc((768,), torch.float32)                      # 3 KB: remembered for offset 0
    ar.reset()
    s = ar.alloc_step((512,), torch.float32)                   # 2 KB at the far end
    again = ar.alloc((768,), torch.float32)                    # the remembered view would run into it
    assert not _overlap(again, s)


def test_finished_parts_are_counted_where_the_parts_lie(monkeypatch):
    """Two step functions (two engines on two streams) never count into the same words, and one step function's counters stay
    where they are (captured steps hold their address); those that a kernel gave up over are set back to zero.  The counters
    that a decode step's launch is given are looked at; nothing is launched."""
    import ctypes
    from types import SimpleNamespace

    from qwen_engine_b200 import ops
    from qwen_engine_b200.engine.runner import ModelRunner
    R, Hq, Hkv, D, P = 12, 16, 8, 128, 16
    ctx_lens, geo, bf = [100 + 150 * i for i in range(R)], (Hq, Hkv, D, 0), torch.bfloat16
    plan = ops.plan_attention([1] * R, ctx_lens, P, (geo,), bf, uniform_splits={geo: ops.TotalParts(37)})
    seen = []

    class Library:
        def __getattr__(self, name):
            def call(*args):
                if name == "qe_decode_attention_mma":
                    seen.append(args[12].value)
                return 0
            return call
    monkeypatch.setattr(ops, "lib", Library)
    monkeypatch.setattr(ops, "_lib", object())
    monkeypatch.setattr(ops, "_ptr", lambda t: ctypes.c_void_p(0 if t is None else t.data_ptr()))
    monkeypatch.setattr(ops, "_stream", lambda: ctypes.c_void_p(0))
    arenas = [Arena("cpu", 1 << 16), Arena("cpu", 1 << 16)]
    for _ in range(2):
        for arena in arenas:
            arena.reset()
            dev = {"plan_" + k: torch.tensor(v, dtype=torch.int32) for k, v in plan.items()}
            ctx = SimpleNamespace(cu_q=torch.arange(R + 1, dtype=torch.int32), ctx_lens=torch.tensor(ctx_lens, dtype=torch.int32),
                                  q_lens_host=[1] * R, ctx_lens_host=ctx_lens, max_q_len=1, arena=arena,
                                  attn_plan=ModelRunner._device_plan(plan, dev, (geo,)))
            ops.paged_attention(torch.zeros(R, (Hq + 2 * Hkv) * D, dtype=bf), torch.zeros(2, 2, Hkv, P, D, dtype=bf),
                                torch.zeros(R, 2, dtype=torch.int32), ctx, torch.zeros(R, Hq * D, dtype=bf), 0.1, 0, Hq, Hkv, D)
    assert len(seen) == 4 and all(seen)
    assert seen[:2] == seen[2:] and seen[0] != seen[1]
    assert all((a.counters["fa"] == 0).all() for a in arenas)
    arenas[1].counters["fa"][5] = 2
    ops.clear_device_status()
    assert (arenas[1].counters["fa"] == 0).all()
