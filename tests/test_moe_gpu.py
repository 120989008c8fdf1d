"""MoE layers on one GPU (world size 1): grouped GEMM with gathered rows, gate-weighted epilogue
and the top-k combine kernel, against a dense PyTorch statement."""
import os

import pytest
import torch
import torch.distributed as dist

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    d = torch.device("cuda", 0)
    if not dist.is_initialized():
        os.environ.setdefault("MASTER_ADDR", "127.0.0.1")
        os.environ.setdefault("MASTER_PORT", "29543")
        dist.init_process_group("nccl", rank=0, world_size=1, device_id=d)
    return d


@pytest.mark.parametrize("tpr,H,ffn,E,topk", [(256, 512, 768, 8, 2), (1000, 256, 384, 16, 4), (64, 128, 256, 4, 1)])
def test_moe_layers_single_gpu(dev, tpr, H, ffn, E, topk):
    from moe_common import run_moe_layer
    run_moe_layer(0, 1, 1, torch.bfloat16, dev, tpr=tpr, H=H, ffn=ffn, E=E, topk=topk, tol=3e-2)


def test_grouped_gemm_plain(dev):
    import tempname_new_b200 as flux
    E, N, K = 6, 384, 256
    splits = torch.tensor([100, 0, 257, 128, 1, 300])
    w = (torch.randn(E, N, K, device=dev) * 0.1).bfloat16()
    x = torch.randn(int(splits.sum()), K, device=dev).bfloat16()
    out = flux.GemmGroupedV3(w, E).forward(x, splits)
    row = 0
    for e, n in enumerate(splits.tolist()):
        ref = x[row:row + n].float() @ w[e].float().t()
        if n:
            assert (out[row:row + n].float() - ref).abs().max().item() <= 2e-2 * max(1.0, ref.abs().max().item())
        row += n


def test_grouped_gemm_fp8_with_scales(dev):
    """e4m3 operands, per-expert weight scale and a scalar input scale applied in the epilogue,
    bf16 output (reference: GemmGroupedV2.forward on 8-bit inputs, src/pybind/gemm_only.cc:171-190)."""
    import tempname_new_b200 as flux
    E, N, K = 5, 512, 384
    splits = torch.tensor([130, 0, 300, 64, 77])
    w = (torch.randn(E, N, K, device=dev) * 0.5).to(torch.float8_e4m3fn)
    x = torch.randn(int(splits.sum()), K, device=dev).to(torch.float8_e4m3fn)
    ws = torch.rand(E, device=dev) + 0.5
    xs = torch.tensor([0.25], device=dev)
    out = flux.GemmGroupedV3(w, E).forward(x, splits, input_scale=xs, weight_scale=ws)
    assert out.dtype == torch.bfloat16
    row = 0
    for e, n in enumerate(splits.tolist()):
        ref = (x[row:row + n].float() @ w[e].float().t()) * ws[e] * 0.25
        if n:
            assert (out[row:row + n].float() - ref).abs().max().item() <= 3e-2 * max(1.0, ref.abs().max().item())
        row += n


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float8_e4m3fn])
def test_moe_layer0_two_weight_groups_share_one_gather(dev, dtype):
    """forward_multiple_weights: gate and up projections on the same gathered rows (the second group
    reads the sorted buffer that the first launch filled)."""
    from moe_common import routed_problem
    import tempname_new_b200 as flux
    tokens, H, ffn, E, topk = 512, 256, 384, 8, 2
    experts, gate, scatter, splits, order = routed_problem(tokens, topk, E, seed=5, device=dev)
    x = (torch.randn(tokens, H, device=dev) * 0.5).to(dtype)
    wg = (torch.randn(E, ffn, H, device=dev) * 0.2).to(dtype)
    wu = (torch.randn(E, ffn, H, device=dev) * 0.2).to(dtype)
    env = flux.DistEnvTPWithEP(dist.group.WORLD, 1, None, ep_size=1)
    op = flux.GemmGroupedV3AGScatter(env, flux.MoeArguments(tokens, H, ffn, E, topk, dtype, torch.bfloat16))
    for _ in range(2):
        og, ou = op.forward_multiple_weights(x, [wg, wu], splits, scatter)
        rows = x[order // topk].float()
        offs = [0] + splits.cumsum(0).tolist()
        for e in range(E):
            lo, hi = offs[e], offs[e + 1]
            if hi > lo:
                for o, w in ((og, wg), (ou, wu)):
                    ref = rows[lo:hi] @ w[e].float().t()
                    assert (o[lo:hi].float() - ref).abs().max().item() <= 3e-2 * max(1.0, ref.abs().max().item())
    op.check_status()


def test_moe_layer1_fused_fp8(dev):
    """The fused combine on e4m3 operands: per-expert weight scales, gate weights per row."""
    from moe_common import routed_problem
    import tempname_new_b200 as flux
    tokens, H, ffn, E, topk = 384, 512, 256, 8, 2
    experts, gate, scatter, splits, order = routed_problem(tokens, topk, E, seed=6, device=dev)
    act = torch.randn(tokens * topk, ffn, device=dev).to(torch.float8_e4m3fn)     # expert-sorted rows
    w2 = (torch.randn(E, H, ffn, device=dev) * 0.3).to(torch.float8_e4m3fn)
    ws = torch.rand(E, device=dev) + 0.5
    row_gate = gate.reshape(-1)[order].contiguous()
    op = flux.GemmGroupedV3GatherRS(E, tokens * topk, H, topk, 0, 1, 1, 1, tp_group=dist.group.WORLD)
    for _ in range(2):
        out = op.forward_gather_rs(act, w2, splits.cpu(), scatter.reshape(-1), weight_scale=ws,
                                   output_vec_scale=row_gate)
        assert out.dtype == torch.bfloat16
        offs = [0] + splits.cumsum(0).tolist()
        y = torch.empty(tokens * topk, H, device=dev)
        for e in range(E):
            lo, hi = offs[e], offs[e + 1]
            y[lo:hi] = (act[lo:hi].float() @ w2[e].float().t()) * ws[e]
        y = (y * row_gate[:, None]).bfloat16().float()
        ref = y[scatter.reshape(-1).long()].view(tokens, topk, H).sum(1)
        assert (out.float() - ref).abs().max().item() <= 3e-2 * max(1.0, ref.abs().max().item())
    op.check_status()


def _gather_case(dev, tokens, E, topk, kind, H, ffn):
    """Layer 0 with two weight groups, twice on one op, against 64 bits; returns the rows per chunk of the gather and what
    the launch with the gather was."""
    import tempname_new_b200 as flux
    from tempname_new_b200 import _native
    g = torch.Generator(device=dev).manual_seed(tokens + E)
    if kind == "random":
        chosen = torch.rand(tokens, E, device=dev, generator=g).topk(topk, dim=1).indices
    elif kind == "one":
        chosen = torch.arange(topk, device=dev).add(E - topk).repeat(tokens, 1)
    else:
        chosen = torch.randint(0, 5, (tokens, topk), device=dev, generator=g) * (E // 5)
    chosen = chosen.to(torch.int32)
    splits, _, scatter, gather, _ = flux.moe_index_build(chosen, E)
    order = torch.argsort(chosen.reshape(-1), stable=True)
    assert torch.equal(gather, (order // topk).int())
    assert torch.equal(splits, torch.bincount(chosen.reshape(-1).long(), minlength=E).int())
    x = torch.randn(tokens, H, device=dev, generator=g).bfloat16()
    w = [(torch.randn(E, ffn, H, device=dev, generator=g) * 0.2).bfloat16() for _ in range(2)]
    env = flux.DistEnvTPWithEP(dist.group.WORLD, 1, None, ep_size=1)
    op = flux.GemmGroupedV3AGScatter(env, flux.MoeArguments(tokens, H, ffn, E, topk, torch.bfloat16, torch.bfloat16))
    rows = x[order // topk].double()
    expert = chosen.reshape(-1)[order].long()
    ref = [torch.empty(tokens * topk, ffn, device=dev, dtype=torch.float64) for _ in range(2)]
    for e in range(E):
        sel = expert == e
        for i in range(2):
            ref[i][sel] = rows[sel] @ w[i][e].double().t()
    for _ in range(2):
        x_now = x.clone()                      # (rows are gathered anew: nothing of the first call may be left over)
        op._sorted = None if op._sorted is None else op._sorted.fill_(float("nan"))
        for got, want in zip(op.forward_multiple_weights(x_now, w, splits, scatter), ref):
            # half a unit in the last place of bf16 is at most 2^-8 of the value; the fp32 sums err by far less
            assert ((got.double() - want).abs() <= 1.01 * 2.0 ** -8 * want.abs() + 2e-6 * H ** 0.5 * want.abs().max()).all()
    op.forward(x, w[0], splits, scatter)
    ran = _native.last_gemm()
    op.check_status()
    warps = 2 * torch.cuda.get_device_properties(dev).multi_processor_count
    return min(max(tokens * topk // (2 * warps), 1), 8), ran


@pytest.mark.parametrize("tokens,E,topk,kind", [(3, 8, 2, "random"), (64, 64, 8, "random"), (64, 64, 1, "one"),
                                                (300, 128, 2, "few"), (4801, 32, 4, "random"), (4801, 8, 4, "one")])
def test_moe_layer0_gather_chunks(dev, tokens, E, topk, kind):
    """Rows are gathered in chunks that may touch several experts (here of one or eight rows), and an expert is
    published when its last row is written: empty experts, one-row experts, all rows on one expert, twice on the same op."""
    chunk, _ = _gather_case(dev, tokens, E, topk, kind, H=136, ffn=128)
    assert chunk == (8 if tokens == 4801 else 1)


@pytest.mark.parametrize("tokens,E,topk,kind,H,ffn,chunk,pair", [
    (4801, 64, 8, "random", 136, 128, 8, 0),       # eight rows per chunk, runs of experts that start anywhere
    (1801, 128, 2, "random", 136, 128, 6, 0),
    (140, 64, 4, "random", 2056, 128, 1, 0),       # rows of 4112 bytes: a whole piece and 16 bytes
    (300, 64, 4, "random", 2056, 128, 2, 0),       # the same, chunks over several experts
    (1500, 512, 2, "random", 2056, 128, 5, 0),
    (1201, 512, 8, "random", 2056, 128, 8, 0),
    (400, 8, 2, "random", 4104, 264, 1, 0),        # two pieces and 16 bytes
    (600, 8, 3, "random", 5000, 128, 3, 0),        # 10000 bytes: two pieces and 1808 bytes
    (1700, 2, 1, "random", 2056, 2048, 2, 1),      # CTA pairs: long rows, chunks over expert boundaries
    (8209, 8, 2, "random", 2056, 2048, 8, 1),
    (13001, 16, 4, "random", 264, 1536, 8, 1),
    (6500, 4, 2, "one", 264, 2048, 8, 1)])
def test_moe_layer0_gather_pieces(dev, tokens, E, topk, kind, H, ffn, chunk, pair):
    """Rows longer than one 4096-byte piece, chunks of up to eight rows that end inside an expert, on single CTAs and
    on CTA pairs."""
    got, ran = _gather_case(dev, tokens, E, topk, kind, H, ffn)
    assert got == chunk
    assert (ran["kernel"], ran["cta_group"], ran["tile_m"]) == (("grouped", 2, 256) if pair else ("grouped", 1, 128))


@pytest.mark.parametrize("n,E", [(1, 1), (31, 512), (511, 64), (513, 8), (4095, 512), (4096, 3), (4097, 64), (20000, 512),
                                 (70001, 7)])
def test_moe_index_build_stable(dev, n, E):
    """The counting sort is stable across lanes, warps and blocks."""
    import tempname_new_b200 as flux
    chosen = torch.randint(0, E, (n,), device=dev, dtype=torch.int32)
    splits, offsets, scatter, gather, tki = flux.moe_index_build(chosen, E)
    order = torch.argsort(chosen, stable=True)
    assert torch.equal(splits.long(), torch.bincount(chosen.long(), minlength=E))
    assert torch.equal(offsets.long(), torch.cat([offsets.new_zeros(1).long(), splits.long().cumsum(0)]))
    assert torch.equal(scatter[order].long(), torch.arange(n, device=dev)) and torch.equal(gather.long(), order)
    assert (tki == 0).all()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float8_e4m3fn])
@pytest.mark.parametrize("splits,N,K", [([1000, 0, 900, 1300], 256, 64), ([769, 768, 1, 1600], 520 + 504, 200),
                                        ([3000, 127, 129, 256], 2056, 144)])
def test_grouped_pairs(dev, dtype, splits, N, K):
    """Tiles shared by two CTAs (768 rows per expert on average and more): one-row and empty experts, tiles whose second
    half has no rows, column and K remainders; contiguous rows, gathered rows and the fused combine."""
    import tempname_new_b200 as flux
    from tempname_new_b200 import _native

    def took_pairs():
        ran = _native.last_gemm()
        return (ran["kernel"], ran["cta_group"], ran["tile_m"], ran["tile_n"]) == ("grouped", 2, 256, 256)

    K = K if dtype.itemsize == 2 else K * 2
    E, rows = len(splits), sum(splits)
    assert rows >= 768 * E
    g = torch.Generator(device=dev).manual_seed(rows + N)
    w = (torch.randn(E, N, K, device=dev, generator=g) * 0.2).to(dtype)
    x = torch.randn(rows, K, device=dev, generator=g).to(dtype)
    expert = torch.repeat_interleave(torch.arange(E, device=dev), torch.tensor(splits, device=dev))
    ref = torch.cat([x[expert == e].float() @ w[e].float().t() for e in range(E)])
    tol = 1e-2 * ref.abs().max().item()
    out = flux.GemmGroupedV3(w, E).forward(x, torch.tensor(splits))
    assert took_pairs()
    assert (out.float() - ref).abs().max().item() <= tol
    # the same rows gathered from shuffled tokens (top-1), and back through the combine
    perm = torch.randperm(rows, device=dev, generator=g)          # token of every sorted row
    tokens = torch.empty_like(x.view(torch.uint8)).view(dtype)
    tokens.view(torch.uint8)[perm] = x.view(torch.uint8)
    scatter = torch.empty(rows, dtype=torch.int32, device=dev)
    scatter[perm] = torch.arange(rows, dtype=torch.int32, device=dev)
    sp = torch.tensor(splits, dtype=torch.int32, device=dev)
    env = flux.DistEnvTPWithEP(dist.group.WORLD, 1, None, ep_size=1)
    o16 = out.dtype
    op = flux.GemmGroupedV3AGScatter(env, flux.MoeArguments(rows, K, N, E, 1, dtype, o16))
    for _ in range(2):
        got = op.forward(tokens, w, sp, scatter.view(rows, 1))
        assert took_pairs()
        assert (got.float() - ref).abs().max().item() <= tol
    op.check_status()
    gate = torch.rand(rows, device=dev, generator=g)
    rs = flux.GemmGroupedV3GatherRS(E, rows, N, 1, 0, 1, 1, 1, tp_group=dist.group.WORLD, dtype=o16)
    for _ in range(2):
        y = rs.forward_gather_rs(x, w, sp, scatter, output_vec_scale=gate)
        assert took_pairs()
        assert (y[perm].float() - ref * gate[:, None]).abs().max().item() <= tol
    rs.check_status()
    # one row less than 768 per expert: single CTAs
    short = torch.tensor([767 * E + E - 1] + [0] * (E - 1))
    flux.GemmGroupedV3(w, E).forward(x.new_zeros(768 * E - 1, K), short)
    assert not took_pairs()


def test_moe_layer0_one_op_unequal_buffers_and_types(dev):
    """One op called with 1-byte rows, then 2-byte rows, the second group's output buffer longer than the first's."""
    from moe_common import routed_problem
    import tempname_new_b200 as flux
    tokens, H, ffn, E, topk = 300, 256, 264, 8, 2
    _, _, scatter, splits, order = routed_problem(tokens, topk, E, seed=5, device=dev)
    env = flux.DistEnvTPWithEP(dist.group.WORLD, 1, None, ep_size=1)
    op = flux.GemmGroupedV3AGScatter(env, flux.MoeArguments(tokens, H, ffn, E, topk, torch.bfloat16, torch.bfloat16))
    expert = torch.repeat_interleave(torch.arange(E, device=dev), splits.long())
    for dtype in (torch.float8_e4m3fn, torch.bfloat16, torch.float8_e4m3fn):
        x = (torch.randn(tokens, H, device=dev) * 0.5).to(dtype)
        ws = [(torch.randn(E, ffn, H, device=dev) * 0.2).to(dtype) for _ in range(2)]
        bufs = [torch.full((tokens * topk + extra, ffn), float("nan"), device=dev, dtype=torch.bfloat16)
                for extra in (0, 500)]
        outs = op.forward_multiple_weights(x, ws, splits, scatter, outputs_buf=bufs)
        rows = x[order // topk].float()
        for out, w in zip(outs, ws):
            ref = torch.cat([rows[expert == e] @ w[e].float().t() for e in range(E)])
            assert (out[:tokens * topk].float() - ref).abs().max().item() <= 1e-2 * ref.abs().max().item()
            assert out[tokens * topk:].isnan().all()
    op.check_status()


@pytest.mark.parametrize("rows", [64, 4096])        # single CTAs; CTA pairs where the rule takes them
def test_grouped_launches_whose_blocks_wait_for_one_another_are_cooperative(dev, rows):
    """The gather and the fused combine need the whole grid resident; a plain grouped GEMM does not."""
    import tempname_new_b200 as flux
    from tempname_new_b200 import _native
    E, H, ffn = 2, 128, 256
    chosen = torch.randint(0, E, (rows, 1), device=dev, dtype=torch.int32)
    splits, _, scatter, _, _ = flux.moe_index_build(chosen, E)
    x, w1, w2 = (torch.randn(*s, device=dev).bfloat16() for s in ((rows, H), (E, ffn, H), (E, H, ffn)))
    env = flux.DistEnvTPWithEP(dist.group.WORLD, 1, None, ep_size=1)
    l0 = flux.GemmGroupedV3AGScatter(env, flux.MoeArguments(rows, H, ffn, E, 1, torch.bfloat16))
    h = l0.forward(x, w1, splits, scatter)
    ran = [_native.last_gemm()]
    flux.GemmGroupedV3GatherRS(E, rows, H, 1, 0, 1, 1, 1, tp_group=dist.group.WORLD).forward_gather_rs(
        h, w2, splits, scatter.reshape(-1))
    ran.append(_native.last_gemm())
    flux.GemmGroupedV3(w1, E).forward(x, splits)
    ran.append(_native.last_gemm())
    assert [r["kernel"] for r in ran] == ["grouped"] * 3
    on = 0 if os.environ.get("FLUXB_COOPERATIVE") == "0" else 1
    assert [r["cooperative"] for r in ran] == [on, on, 0]
