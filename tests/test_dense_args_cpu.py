"""The tile choices of the dense kernel and what the ops hand to its launcher, on the CPU."""
import pytest
import torch
import torch.distributed as dist
from torch.autograd import forward_ad

from conftest import free_port, run_gloo
from fake_launch import Recorder, as_cuda, record_launches
from tempname_new_b200.tuning import table


def _several_ranks(m, n, k):
    """The choices that the fused ops of several ranks were measured with."""
    if (m, n, k) in ((4096, 4096, 4096), (4096, 12288, 4096), (16384, 8192, 3584)):
        return {"cta_group": 2, "tile_n": 256, "tile_m": 512, "group_m": 8}
    if m >= 256 and n >= 256 and (m // 256) * -(-n // 256) >= 37:
        return {"cta_group": 2, "tile_n": 256, "group_m": 8}
    return {"cta_group": 1, "tile_n": 256 if n % 256 == 0 or n > 2048 else 128, "group_m": 16}


@pytest.mark.parametrize("ranks", [2, 4, 8])
def test_tile_choices_of_several_ranks(ranks):
    for m in (64, 256, 300, 1000, 1024, 2048, 4096, 8192, 16384, 32768):
        for n in (128, 264, 1024, 3000, 4096, 8192, 12288):
            for k in (256, 3584, 4096, 5120, 12288):
                if (m, n, k) not in table.DENSE_TABLE:
                    for elt in (1, 2):
                        assert table.lookup(m, n, k, elt, ranks) == _several_ranks(m, n, k)
    assert table.lookup(8192, 12288, 49152, 2, ranks)["group_m"] == 4


def _landing_buffer(rank, world):
    import tempname_new_b200 as flux
    rec = record_launches()
    M, N, K = 512, 256, 256
    op = flux.AGKernel(dist.group.WORLD, 1, M, N, K, torch.float8_e4m3fn)
    op.status = torch.zeros(4, dtype=torch.int32)
    for dtype, rows, fits in ((torch.float8_e4m3fn, M, True), (torch.bfloat16, M, False), (torch.bfloat16, M // 2, True)):
        x, w = (as_cuda(torch.zeros(r, K).to(dtype)) for r in (rows // world, N))
        before = len(rec.calls)
        if fits:
            op.forward(x, w)
        else:
            with pytest.raises(ValueError, match="landing buffer"):
                op.forward(x, w)
        assert len(rec.calls) == before + fits


def test_all_gather_push_stays_inside_the_landing_buffers():
    run_gloo(_landing_buffer, 2)


def _rank_counts(rank, world):
    import tempname_new_b200 as flux
    rec = record_launches()
    pg, status, bf = dist.group.WORLD, torch.zeros(4, dtype=torch.int32), torch.bfloat16
    M, N, K = 2048, 4096, 1024              # a short K: one rank alone would take bands of 16 tile rows
    seen = table.lookup(M, N, K), table.lookup(M, N, K, 2, world)
    assert seen[0]["group_m"] == 16 and seen[1]["group_m"] == 8
    x, w = as_cuda(torch.zeros(M, K, dtype=bf)), as_cuda(torch.zeros(N, K, dtype=bf))
    rs = flux.GemmRS(pg, 1, M, N, bf)
    ag = flux.AGKernel(pg, 1, M, N, K, bf)
    pre = flux.GemmAllToAllTranspose(pg, 1, world, 1, M * world, K, 64, N, bf)
    post = flux.AllToAllTransposeGemm(pg, 1, world, 1, K // 64, M * world, 64, bf)
    for op in (rs, ag, pre, post):
        op.status = status
    post.land.view = lambda r, dtype, shape: as_cuda(torch.zeros(shape, dtype=dtype))
    rs.forward(x, w)
    ag.forward(x[:M // world], w)
    pre.forward(x.view(1, M, K), w)
    post.forward(as_cuda(torch.zeros(1, K // 64 // world, M * world, 64, dtype=bf)), w)
    assert len(rec.calls) == 4
    for a in rec.calls:
        b = getattr(a, "base", a)
        assert (b.cta_group, b.tile_n, b.group_m) == (2, 256, 8)


def test_fused_ops_ask_for_their_rank_count():
    run_gloo(_rank_counts, 2)


@pytest.fixture
def row_parallel(monkeypatch):
    """A row-parallel layer of one rank that takes the CUDA branch, its input, and the recorder."""
    from tempname_new_b200 import _native
    from tempname_new_b200.ops import _dense
    from tempname_new_b200.parallel.layers import RowParallelLinear
    created = not dist.is_initialized()
    if created:
        dist.init_process_group("gloo", init_method=f"tcp://127.0.0.1:{free_port()}", rank=0, world_size=1)
    rec = Recorder(_native.lib())
    monkeypatch.setattr(_native, "lib", lambda: rec)
    monkeypatch.setattr(_dense, "current_stream_ptr", lambda device=None: 0)
    lin = RowParallelLinear(64, 128)
    lin.requires_grad_(False)
    lin.weight = torch.nn.Parameter(as_cuda(lin.weight.data), requires_grad=False)
    lin._cache.rs(32, 128, torch.bfloat16).status = torch.zeros(4, dtype=torch.int32)
    yield lin, as_cuda(torch.zeros(32, 64, dtype=torch.bfloat16)), rec
    lin._cache.ops.clear()
    if created:
        dist.destroy_process_group()


def test_row_parallel_bias_with_a_forward_mode_tangent(row_parallel):
    lin, x, rec = row_parallel
    lin(x)
    assert rec.calls[-1].bias == lin.bias.data_ptr()
    bias = lin.bias.detach()
    tangent = torch.randn(128).bfloat16()
    del lin.bias
    with forward_ad.dual_level():
        lin.bias = forward_ad.make_dual(bias, tangent)
        y = lin(x)
        assert rec.calls[-1].bias is None
        assert torch.equal(forward_ad.unpack_dual(y).tangent, tangent.expand(32, 128))


@pytest.mark.parametrize("shape", [(1, 128), (1,), (), (32, 128)])
def test_row_parallel_bias_that_broadcasts(row_parallel, shape):
    """A bias of another shape than [out] is added as PyTorch broadcasts it, and gets a gradient of its shape."""
    lin, x, rec = row_parallel
    lin.bias = torch.nn.Parameter(torch.randn(shape).bfloat16())
    x.requires_grad_(True)
    y = lin(x)
    assert rec.calls[-1].bias is None and y.shape == (32, 128)
    (g,) = torch.autograd.grad(y, [lin.bias], torch.ones(32, 128).bfloat16())
    assert g.shape == shape and torch.equal(g, torch.full(shape, 32 * 128 / max(1, lin.bias.numel())).bfloat16())


@pytest.mark.parametrize("M,N,k_blocks,rule", [
    (128, 16384, 32, (64, 256, 1)), (2048, 1024, 48, (64, 256, 1)),       # 64 columns fill the chip without a split
    (128, 16384, 49, (128, 128, 2)), (2048, 1024, 64, (128, 128, 2)),     # a long K: two halves of 128 columns
    (128, 4096, 48, (64, 64, 2)), (128, 4096, 64, (64, 64, 4)), (64, 16384, 32, (128, 128, 2)), (128, 32768, 32, (0, 0, 0))])
def test_split_k_tiles(M, N, k_blocks, rule):
    """(columns, tiles, CTAs per tile) on both sides of the lines, for 148 SMs."""
    import ctypes
    from tempname_new_b200 import _native
    v = [ctypes.c_int32() for _ in range(3)]
    _native.check(_native.lib().fluxb_skinny_shape(M, N, k_blocks, 0, 148, *map(ctypes.byref, v)), "rule")
    assert tuple(x.value for x in v) == rule
