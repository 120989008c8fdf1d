"""What the MoE layer-0 op hands to its kernel, on the CPU."""
import pytest
import torch
import torch.distributed as dist

from conftest import free_port, run_gloo
from fake_launch import Recorder, as_cuda, record_launches
from moe_common import routed_problem


@pytest.fixture
def layer0(monkeypatch):
    """(tokens, hidden, ffn, experts, topk, dtype) -> (op, recorder, routing of the tokens)."""
    import tempname_new_b200 as flux
    from tempname_new_b200 import _native
    from tempname_new_b200.ops import _dense
    monkeypatch.delenv("FLUXB_MOE_GATHER", raising=False)
    created = not dist.is_initialized()
    if created:
        dist.init_process_group("gloo", init_method=f"tcp://127.0.0.1:{free_port()}", rank=0, world_size=1)
    rec = Recorder(_native.lib())
    monkeypatch.setattr(_native, "lib", lambda: rec)
    monkeypatch.setattr(_dense, "current_stream_ptr", lambda device=None: 0)

    def make(tokens, H, ffn, E, topk, dtype):
        env = flux.DistEnvTPWithEP(dist.group.WORLD, 1, None, ep_size=1)
        op = flux.GemmGroupedV3AGScatter(env, flux.MoeArguments(tokens, H, ffn, E, topk, dtype, torch.bfloat16))
        op.status = torch.zeros(4, dtype=torch.int32)
        _, _, scatter, splits, _ = routed_problem(tokens, topk, E)
        return op, rec, splits, scatter

    yield make
    if created:
        dist.destroy_process_group()


def test_sorted_rows_buffer_follows_the_element_type(layer0):
    """The gather writes rows of the call's element type into the sorted buffer: one kept from a call with 1-byte rows
    is half the size that a call with 2-byte rows of the same count writes."""
    tokens, H, ffn, E, topk = 256, 64, 128, 4, 2
    op, rec, splits, scatter = layer0(tokens, H, ffn, E, topk, torch.bfloat16)
    for dtype in (torch.float8_e4m3fn, torch.bfloat16, torch.float8_e4m3fn):
        x = as_cuda(torch.zeros(tokens, H).to(dtype))
        op.forward(x, torch.zeros(E, ffn, H).to(dtype), splits, scatter)
        a = rec.calls[-1]
        assert a.a_sorted == op._sorted.data_ptr() and a.a_sorted_rows >= tokens * topk
        assert op._sorted.numel() * op._sorted.element_size() >= a.a_sorted_rows * H * dtype.itemsize
        assert op._sorted.dtype == dtype


def test_weight_groups_share_one_sorted_rows_buffer(layer0):
    """Groups after the first read the rows that the first one gathered, also when their output buffer is longer."""
    tokens, H, ffn, E, topk = 256, 64, 128, 4, 2
    op, rec, splits, scatter = layer0(tokens, H, ffn, E, topk, torch.bfloat16)
    x = as_cuda(torch.zeros(tokens, H).bfloat16())
    w = torch.zeros(E, ffn, H).bfloat16()
    bufs = [torch.empty(n, ffn).bfloat16() for n in (tokens * topk, tokens * topk + 300, tokens * topk)]
    op.forward_multiple_weights(x, [w, w, w], splits, scatter, outputs_buf=bufs)
    first, *rest = rec.calls
    assert first.gathered == 1 and first.a_sorted_rows >= tokens * topk + 300
    assert [(a.gathered, a.a, a.reuse_schedule) for a in rest] == [(0, first.a_sorted, 1)] * 2


def test_combine_slots_hold_sixteen_bit_rows(layer0):
    """An op built for 8-bit inputs receives 16-bit rows in its staging slots, like any other."""
    import tempname_new_b200 as flux
    tokens, H, E, topk = 64, 256, 4, 2
    layer0(tokens, H, 128, E, topk, torch.bfloat16)
    for dtype in (torch.bfloat16, torch.float8_e4m3fn, torch.float8_e5m2):
        op = flux.GemmGroupedV3GatherRS(E, tokens * topk, H, topk, 0, 1, 1, 1, tp_group=dist.group.WORLD, dtype=dtype)
        assert op.stage.nbytes >= tokens * topk * H * 2


def _landing_buffer(rank, world):
    import tempname_new_b200 as flux
    tokens, H, ffn, E, topk = 128, 64, 128, 4, 2          # (of all ranks)
    env = flux.DistEnvTPWithEP(dist.group.WORLD, 1, None, ep_size=world)
    op = flux.GemmGroupedV3AGScatter(env, flux.MoeArguments(tokens, H, ffn, E, topk, torch.float8_e4m3fn))
    op.status = torch.zeros(4, dtype=torch.int32)
    rec = record_launches()
    _, _, scatter, splits, _ = routed_problem(tokens, topk, E)
    for dtype, hidden, fits in ((torch.float8_e4m3fn, H, True), (torch.bfloat16, H, False),
                                (torch.bfloat16, H // 2, True), (torch.float8_e4m3fn, 2 * H, False)):
        x = as_cuda(torch.zeros(tokens // world, hidden).to(dtype))
        w = torch.zeros(E // world, ffn, hidden).to(dtype)
        before = len(rec.calls)
        if fits:
            op.forward(x, w, splits, scatter)
        else:
            with pytest.raises(ValueError, match="landing buffer"):
                op.forward(x, w, splits, scatter)
        assert len(rec.calls) == before + fits


def test_token_push_stays_inside_the_landing_buffers():
    """Several ranks: tokens wider than the landing buffers were made for are refused, not written past their end."""
    run_gloo(_landing_buffer, 2)


def _many_experts(rank, world):
    import tempname_new_b200 as flux
    tokens, H, ffn, topk = 128, 64, 128, 2
    rec = record_launches()
    for E, first_gathers in ((256, True), (512, False)):
        env = flux.DistEnvTPWithEP(dist.group.WORLD, 1, None, ep_size=1)
        op = flux.GemmGroupedV3AGScatter(env, flux.MoeArguments(tokens, H, ffn * world, E, topk, torch.bfloat16))
        op.status = torch.zeros(4, dtype=torch.int32)
        _, _, scatter, splits, _ = routed_problem(tokens, topk, E)
        w = torch.zeros(E, ffn, H).bfloat16()
        del rec.calls[:]
        op.forward_multiple_weights(as_cuda(torch.zeros(tokens // world, H).bfloat16()), [w, w, w], splits, scatter)
        # 512 experts from two sources: the first launch gathers in the loader, the second fills the buffer
        assert [a.gathered for a in rec.calls] == ([1, 0, 0] if first_gathers else [1, 1, 0])
        assert [a.do_allgather for a in rec.calls] == [1, 0, 0]


def test_sorted_rows_are_reused_only_where_a_launch_filled_them():
    run_gloo(_many_experts, 2)
