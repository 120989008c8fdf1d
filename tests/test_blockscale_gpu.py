"""Block-scaled fp8 GEMM on the GPU against the PyTorch statement of the op."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    return torch.device("cuda", 0)


def _quantized(M, N, K, dev, seed=0):
    import tempname_new_b200 as flux
    g = torch.Generator(device=dev).manual_seed(seed)
    x = torch.randn(M, K, device=dev, generator=g).bfloat16()
    w = (torch.randn(N, K, device=dev, generator=g) * 0.05).bfloat16()
    # make block scales differ a lot so that a wrong scale index shows
    x[: M // 2] *= 8
    w[:, K // 2:] *= 0.1
    qz = flux.Quantization(torch.bfloat16, torch.float8_e4m3fn)
    xq, sx, _, _ = qz.quantize_vector_blockwise(x, False)
    wq, sw, _, _ = qz.quantize_square_blockwise(w, False)
    return x, w, xq, sx, wq, sw


@pytest.mark.parametrize("M,N,K", [(128, 128, 128), (256, 384, 512), (512, 1024, 2048), (1024, 3584, 8192),
                                   (384, 2176, 640)])   # 128 x 256 tiles with a half-empty last column tile
def test_blockscale_gemm(dev, M, N, K):
    import tempname_new_b200 as flux
    x, w, xq, sx, wq, sw = _quantized(M, N, K, dev)
    op = flux.BlockScaleGemm(torch.float8_e4m3fn, torch.float8_e4m3fn, torch.bfloat16)
    out = op.forward(xq, wq, input_scale=sx, weight_scale=sw)
    ref = flux.blockscale_gemm_torch(xq, wq, sx, sw, torch.float32)
    full = x.float() @ w.float().t()
    tol = 2e-2 * max(1.0, ref.abs().max().item())
    assert (out.float() - ref).abs().max().item() <= tol
    # and the quantised product tracks the unquantised one
    rel = (out.float() - full).norm() / full.norm()
    assert rel.item() < 0.06


def test_blockscale_bias_and_grouped(dev):
    import tempname_new_b200 as flux
    M, N, K, E = 512, 256, 512, 2
    x, w, xq, sx, wq, sw = _quantized(M, N * E, K, dev, seed=1)
    op = flux.BlockScaleGemm()
    bias = torch.randn(N * E, device=dev).bfloat16()
    out = op.forward(xq, wq, bias=bias, input_scale=sx, weight_scale=sw)
    ref = flux.blockscale_gemm_torch(xq, wq, sx, sw, torch.float32, bias)
    assert (out.float() - ref).abs().max().item() <= 2e-2 * max(1.0, ref.abs().max().item())
    wq3, sw3 = wq.view(E, N, K), sw.view(E, N // 128, K // 128)
    outg = op.forward_grouped(xq, torch.tensor([256, 256]), wq3, input_scale=sx, weight_scale=sw3)
    # the same on one stream must give the same bits
    one = flux.BlockScaleGemm(num_streams=1).forward_multi_stream(xq, [256, 256], wq3, input_scale=sx, weight_scale=sw3)
    assert torch.equal(outg, one)
    for e in range(E):
        r = flux.blockscale_gemm_torch(xq[e * 256:(e + 1) * 256], wq3[e], sx[e * 2:(e + 1) * 2], sw3[e], torch.float32)
        assert (outg[e * 256:(e + 1) * 256].float() - r).abs().max().item() <= 2e-2 * max(1.0, r.abs().max().item())


def test_blockscale_per_expert_forms_on_side_streams(dev):
    """Experts of different sizes (one empty) dealt over three side streams, called twice in a row and
    followed at once by work on the caller's stream: the join must order it after every expert."""
    import tempname_new_b200 as flux
    N, K, E = 256, 512, 5
    splits = [128, 384, 0, 256, 640]
    M = sum(splits)
    x, w, xq, sx, wq, sw = _quantized(M, N * E, K, dev, seed=3)
    wq3, sw3 = wq.view(E, N, K), sw.view(E, N // 128, K // 128)
    op = flux.BlockScaleGemm(num_streams=3)
    for _ in range(2):
        out = op.forward_multi_stream(xq, splits, wq3, input_scale=sx, weight_scale=sw3)
        total = out.float().sum()                       # the caller's stream reads the result right away
    row = 0
    ref_total = 0.0
    for e, cnt in enumerate(splits):
        if cnt:
            r = flux.blockscale_gemm_torch(xq[row:row + cnt], wq3[e], sx[row // 128:(row + cnt) // 128], sw3[e],
                                           torch.float32)
            assert (out[row:row + cnt].float() - r).abs().max().item() <= 2e-2 * max(1.0, r.abs().max().item())
            ref_total += out[row:row + cnt].float().sum().item()
        row += cnt
    assert abs(total.item() - ref_total) <= 1e-3 * max(1.0, abs(ref_total))


@pytest.mark.parametrize("M,N,K", [(256, 384, 512), (1024, 1024, 1024),
                                   (128, 256, 128),        # one k-block: nothing to fetch ahead
                                   (200, 2176, 384),       # ragged rows, odd k-blocks, half-empty last column tile
                                   (19 * 128, 2304, 640)])  # more tiles than CTAs: buffers change parity per tile
def test_blockscale_wgrad_form_per_column_weight_scales(dev, M, N, K):
    """Both operands carry 1x128 scales (weight_scale [N/128, K/128, 128]): the weight-gradient form,
    on the kernel, against the PyTorch statement."""
    import tempname_new_b200 as flux
    x, w, xq, sx, _, _ = _quantized(M, N, K, dev, seed=2)
    qz = flux.Quantization(torch.bfloat16, torch.float8_e4m3fn)
    wq, sw, _, _ = qz.quantize_vector_blockwise(w, False)           # 1x128 scales for the weight rows too
    assert tuple(sw.shape) == (N // 128, K // 128, 128)
    op = flux.BlockScaleGemm()
    out = op.wgrad(xq, wq, input_scale=sx, weight_scale=sw)
    ref = flux.blockscale_gemm_torch(xq, wq, sx, sw, torch.float32)
    assert (out.float() - ref).abs().max().item() <= 2e-2 * max(1.0, ref.abs().max().item())


def test_blockscale_ragged_rows(dev):
    """M that is not a multiple of 128: the last row block is partial (its scales exist, rows clipped)."""
    import tempname_new_b200 as flux
    M, N, K = 300, 256, 512
    x, w, xq, sx, wq, sw = _quantized(M, N, K, dev, seed=3)
    assert sx.shape[0] == 3
    out = flux.BlockScaleGemm().forward(xq, wq, input_scale=sx, weight_scale=sw)
    ref = flux.blockscale_gemm_torch(xq, wq, sx, sw, torch.float32)
    assert out.shape == (M, N)
    assert (out.float() - ref).abs().max().item() <= 2e-2 * max(1.0, ref.abs().max().item())


@pytest.mark.parametrize("M,N,K", [(1, 128, 128), (7, 512, 256), (48, 3584, 8192), (128, 8192, 512), (200, 8192, 1152),
                                   (1000, 2048, 2048), (64, 16384, 640)])
def test_split_k_block_scaled(dev, M, N, K):
    """The split-K form against 64 bits and against the persistent kernel: partial row blocks, one to four splits."""
    from tempname_new_b200 import _native
    from tempname_new_b200.ops import _dense
    from tempname_new_b200.ops.blockscale_gemm import blockscale_args
    import tempname_new_b200 as flux
    g = torch.Generator(device=dev).manual_seed(M + N + K)
    a, b = (torch.randn(s, device=dev, generator=g).to(torch.float8_e4m3fn) for s in ((M, K), (N, K)))
    sa = torch.rand((M + 127) // 128, K // 128, 128, device=dev, generator=g) + 0.5
    sb = torch.rand(N // 128, K // 128, device=dev, generator=g) + 0.5
    bias = torch.randn(N, device=dev, generator=g).bfloat16()
    ad = a.double().view(M, K // 128, 128) * sa.double().permute(0, 2, 1).reshape(-1, K // 128)[:M, :, None]
    bd = b.double().view(N, K // 128, 128) * sb.double().repeat_interleave(128, 0)[:, :, None]
    ref = ad.reshape(M, K) @ bd.reshape(N, K).t() + bias.double()
    new = flux.BlockScaleGemm().forward(a, b, bias=bias, input_scale=sa, weight_scale=sb)
    assert _native.last_gemm()["kernel"] == "split_k"
    old = torch.empty(M, N, device=dev, dtype=torch.bfloat16)
    args = blockscale_args(a, b, sa, sb, bias, torch.bfloat16, M)
    args.auto_shape, args.tile_n, args.M, args.d, args.ldd = 0, 128, M, old.data_ptr(), N
    args.mode, args.rank, args.world, args.epoch = _dense.PLAIN, 0, 1, 1
    _dense.run(args)
    assert _native.last_gemm()["kernel"] == "persistent"
    e_new, e_old = ((t.double() - ref).norm().item() for t in (new, old))
    assert not new.isnan().any() and e_new <= 1.02 * e_old and e_new <= 2e-3 * ref.norm().item()


@pytest.mark.parametrize("M,N,K", [(200, 2176, 384), (128, 256, 128), (2432, 2304, 640), (1184, 4224, 256),
                                   (2500, 1792, 512), (2500, 1920, 512)])
@pytest.mark.parametrize("groupwise", [False, True])
def test_cut_tiles_of_the_last_wave(dev, M, N, K, groupwise):
    """128 x 256 tiles whose last wave is cut into 128-column halves (all tiles, some, none; a half past the last column),
    with one weight scale per block, and the same problems with one per column, whose tiles stay whole: against 64 bits,
    and bit for bit against whole 128 x 128 tiles, which multiply and add in the same order."""
    from tempname_new_b200 import _native
    from tempname_new_b200.ops import _dense
    from tempname_new_b200.ops.blockscale_gemm import blockscale_args
    g = torch.Generator(device=dev).manual_seed(M + N + K)
    a, b = (torch.randn(s, device=dev, generator=g).to(torch.float8_e4m3fn) for s in ((M, K), (N, K)))
    sa = torch.rand((M + 127) // 128, K // 128, 128, device=dev, generator=g) + 0.5
    sb = torch.rand(*((N // 128, K // 128) + ((128,) if groupwise else ())), device=dev, generator=g) + 0.5
    ad = a.double().view(M, K // 128, 128) * sa.double().permute(0, 2, 1).reshape(-1, K // 128)[:M, :, None]
    sbd = sb.double().permute(0, 2, 1).reshape(N, K // 128) if groupwise else sb.double().repeat_interleave(128, 0)
    ref = ad.reshape(M, K) @ (b.double().view(N, K // 128, 128) * sbd[:, :, None]).reshape(N, K).t()
    outs = []
    for tile_n in (256, 128):
        out = torch.full((M, N), float("nan"), device=dev, dtype=torch.bfloat16)
        args = blockscale_args(a, b, sa, sb, None, torch.bfloat16, M)
        args.auto_shape, args.tile_n, args.M, args.d, args.ldd = 0, tile_n, M, out.data_ptr(), N
        args.mode, args.rank, args.world, args.epoch = _dense.PLAIN, 0, 1, 1
        _dense.run(args)
        ran = _native.last_gemm()
        wide = tile_n == 256 and N != 1920         # (an odd number of 128-column blocks below 2048: narrow tiles)
        cut = 2 if wide and not groupwise and M != 2500 else 1
        assert (ran["kernel"], ran["tile_n"], ran["splits"]) == ("persistent", 256 if wide else 128, cut)
        assert (out.double() - ref).norm().item() <= 2e-3 * ref.norm().item()
        outs.append(out)
    assert torch.equal(*outs)
