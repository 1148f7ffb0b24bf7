"""GPU parity of the fused linear layer (C ABI: hdit_linear_fused) against an fp32 torch restatement of what the
reference runs unfused: torch.nn.Linear (one rounding to 16 bits), then the eager GELU or gated residual
(layers/feedforward.py:73-78 and the residual additions around layers/attention_processor.py:207-449).

Tolerance for 16-bit activations: cosine >= 0.9999 and max|a - b| / max|b| <= 2e-2 per case."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _want(x, w, b, epilogue, residual=None, gate=None):
    y = F.linear(x.float(), w.float(), b.float() if b is not None else None).to(x.dtype).float()
    if epilogue == "gelu_tanh":
        y = F.gelu(y, approximate="tanh")
    elif epilogue == "gate_residual":
        y = residual.float() + gate.float()[:, None, :] * y
    return y.to(x.dtype)


def _check(got, want):
    g, w = got.float().flatten(), want.float().flatten()
    assert torch.isfinite(g).all()
    cos = F.cosine_similarity(g, w, dim=0).item()
    rel = ((g - w).abs().max() / w.abs().max().clamp_min(1e-6)).item()
    assert cos >= 0.9999 and rel <= 2e-2, (cos, rel)


def _inputs(B, S, K, N, dtype, seed):
    gen = torch.Generator().manual_seed(seed)
    x = torch.randn(B, S, K, generator=gen).to(dtype).to(DEV)
    w = (torch.randn(N, K, generator=gen) / K ** 0.5).to(dtype).to(DEV)
    b = torch.randn(N, generator=gen).to(dtype).to(DEV)
    res = torch.randn(B, S, N, generator=gen).to(dtype).to(DEV)
    gate = torch.randn(B, N, generator=gen).to(dtype).to(DEV)
    return x, w, b, res, gate


# (tile_m, tile_n, cta_pair): 0 = the library chooses; cta_pair 2 = two CTAs share a 256 x 256 tile
TILES = [(0, 0, 0), (128, 128, 1), (128, 256, 1), (256, 256, 1), (0, 0, 2)]


@pytest.mark.parametrize("epilogue", ["bias", "gelu_tanh", "gate_residual"])
@pytest.mark.parametrize("tile", TILES, ids=lambda t: f"tile{t[0]}x{t[1]}pair{t[2]}")
@pytest.mark.parametrize("B,S,K,N", [(1, 128, 64, 256), (1, 300, 200, 264), (2, 333, 1024, 1160), (1, 576, 3072, 3072)])
def test_linear_fused_matches_unfused_chain(B, S, K, N, tile, epilogue):
    from hetu_dit_b200 import kernels
    x, w, b, res, gate = _inputs(B, S, K, N, torch.bfloat16, B * 1000 + S + K + N)
    got = kernels.linear_fused(x, w, b, epilogue=epilogue, residual=res, gate=gate, tile_m=tile[0], tile_n=tile[1],
                               cta_pair=tile[2])
    torch.cuda.synchronize()
    _check(got, _want(x, w, b, epilogue, res, gate))


def test_linear_fused_many_tiles_per_cta_and_long_k():
    """Few persistent CTAs walk many tiles: both accumulators and every ring stage are re-used many times."""
    from hetu_dit_b200 import kernels
    x, w, b, res, gate = _inputs(1, 1100, 4160, 1544, torch.bfloat16, 7)
    for tile_m, tile_n, pair in TILES[1:]:
        for ctas in (2, 3, 7):
            got = kernels.linear_fused(x, w, b, epilogue="gate_residual", residual=res, gate=gate, tile_m=tile_m,
                                       tile_n=tile_n, max_ctas=ctas, cta_pair=pair)
            torch.cuda.synchronize()
            _check(got, _want(x, w, b, "gate_residual", res, gate))


def test_linear_fused_fp16_no_bias_strided_and_in_place():
    from hetu_dit_b200 import kernels
    x, w, b, res, gate = _inputs(2, 200, 512, 384, torch.float16, 11)
    for pair in (1, 2):
        got = kernels.linear_fused(x, w, None, epilogue="bias", cta_pair=pair)
        _check(got, _want(x, w, None, "bias"))
    # the result lands in a column block of a wider buffer; rows of x are a column block too
    wide_in = torch.zeros(2, 200, 512 + 64, dtype=torch.float16, device=DEV)
    wide_in[..., 64:] = x
    wide_out = torch.full((2, 200, 1024), 7.0, dtype=torch.float16, device=DEV)
    kernels.linear_fused(wide_in[..., 64:], w, b, epilogue="gelu_tanh", out=wide_out[..., 128:128 + 384])
    torch.cuda.synchronize()
    _check(wide_out[..., 128:128 + 384], _want(x, w, b, "gelu_tanh"))
    assert (wide_out[..., :128] == 7.0).all() and (wide_out[..., 128 + 384:] == 7.0).all()
    # out aliases the residual
    want = _want(x, w, b, "gate_residual", res, gate)
    kernels.linear_fused(x, w, b, epilogue="gate_residual", residual=res, gate=gate, out=res)
    torch.cuda.synchronize()
    _check(res, want)


def test_linear_fused_two_dim_and_argument_errors():
    from hetu_dit_b200 import _C, kernels
    x, w, b, _, _ = _inputs(1, 130, 128, 136, torch.bfloat16, 13)
    got = kernels.linear_fused(x[0], w, b)
    torch.cuda.synchronize()
    _check(got, _want(x, w, b, "bias")[0])
    with pytest.raises(_C.HditError):
        kernels.linear_fused(x[..., :60], w[:, :60].contiguous(), b)  # k not a multiple of 8
    with pytest.raises(_C.HditError):
        kernels.linear_fused(x, w, b, tile_n=64)
    with pytest.raises(_C.HditError):
        kernels.linear_fused(x, w, b, tile_n=128, cta_pair=2)
    with pytest.raises(ValueError):
        kernels.linear_fused(x, w[:, :64], b)


def test_linear_fused_flux_mlp_shapes():
    """The shapes of one Flux single block at full size: (4608, 3072) x (12288, 3072)^T with GELU, then
    (4608, 15360) x (3072, 15360)^T with the gated residual; checked on a row subset."""
    from hetu_dit_b200 import kernels
    gen = torch.Generator(device=DEV).manual_seed(5)
    d = 3072
    x = torch.randn(1, 4608, d, device=DEV, generator=gen).to(torch.bfloat16)
    w1 = (torch.randn(4 * d, d, device=DEV, generator=gen) / d ** 0.5).to(torch.bfloat16)
    b1 = torch.randn(4 * d, device=DEV, generator=gen).to(torch.bfloat16)
    w2 = (torch.randn(d, 5 * d, device=DEV, generator=gen) / (5 * d) ** 0.5).to(torch.bfloat16)
    b2 = torch.randn(d, device=DEV, generator=gen).to(torch.bfloat16)
    gate = torch.randn(1, d, device=DEV, generator=gen).to(torch.bfloat16)
    buf = torch.randn(1, 4608, 5 * d, device=DEV, generator=gen).to(torch.bfloat16)
    rows = torch.arange(0, 4608, 37, device=DEV)
    for pair in (1, 2):
        buf[..., d:].zero_()
        kernels.linear_fused(x, w1, b1, epilogue="gelu_tanh", out=buf[..., d:], cta_pair=pair)
        out = kernels.linear_fused(buf, w2, b2, epilogue="gate_residual", residual=x, gate=gate, cta_pair=pair)
        torch.cuda.synchronize()
        _check(buf[:, rows, d:], _want(x[:, rows], w1, b1, "gelu_tanh"))
        _check(out[:, rows], _want(buf[:, rows], w2, b2, "gate_residual", x[:, rows], gate))


def _group_case(D, norm, rope, S, B, dtype, seed, H=6, K=328):
    gen = torch.Generator().manual_seed(seed)
    lin = torch.nn.Linear(K, H * D, device=DEV, dtype=dtype)
    with torch.no_grad():
        lin.weight.copy_(torch.randn(H * D, K, generator=gen) / K ** 0.5)
        lin.bias.copy_(torch.randn(H * D, generator=gen))
    x = torch.randn(B, S, K, generator=gen).to(dtype).to(DEV)
    w = (1 + 0.2 * torch.randn(D, generator=gen)).to(dtype).to(DEV) if norm else None
    b = (0.2 * torch.randn(D, generator=gen)).to(dtype).to(DEV) if norm == 2 else None
    return lin, x, (norm, w, b, 1e-6) if norm else None, rope


# (head_dim, norm kind, (rope_seq_start, rope_row0) or None, rows per batch entry, batch): rows around the 32-row slices,
# the 128- and 256-row tiles, batch entries that end inside a slice, rotation that starts inside a tile
NORM_ROPE = [(128, 1, (0, 0), 1, 1), (128, 1, (0, 3), 257, 1), (64, 1, None, 127, 2), (64, 2, (17, 0), 129, 2),
             (64, 2, (0, 5), 33, 5), (128, 0, (40, 0), 300, 1), (64, 0, (0, 0), 256, 1), (128, 1, (31, 1), 96, 3)]


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("tile", TILES, ids=lambda t: f"tile{t[0]}x{t[1]}pair{t[2]}")
@pytest.mark.parametrize("D,norm,rope,S,B", NORM_ROPE)
def test_linear_group_norm_rope_is_the_linear_layer_then_qk_norm_rope(D, norm, rope, S, B, tile, dtype):
    """Same accumulators, same rounding points and order of sums: the bits of the two launches it replaces. The second
    item (another row count) has no norm; the third writes rows in the middle of a wider buffer."""
    from hetu_dit_b200 import _C, kernels
    lin, x, nrm, rp = _group_case(D, norm, rope, S, B, dtype, 100 * D + S)
    lin2, x2, _, _ = _group_case(D, 0, None, 77, 1, dtype, 5)
    gen = torch.Generator().manual_seed(3)
    rows = S + 8
    cos, sin = (torch.randn(rows, D, generator=gen).to(DEV) for _ in range(2))
    kw = dict(tile_m=tile[0], tile_n=tile[1], cta_pair=tile[2])
    wide = torch.full((B, S, 6 * D + 64), 3.0, dtype=dtype, device=DEV)
    with torch.no_grad():
        got, got2, got3 = kernels.linear_group(
            [kernels.Lin(x, lin, "norm_rope", head_dim=D, norm=nrm, rope=rp), kernels.Lin(x2, lin2),
             kernels.Lin(x, lin, "gelu_tanh", out=wide[..., 64:])], cos, sin, **kw)
        plain = kernels.linear_fused(x, lin.weight, lin.bias, **kw)
        want = plain.clone().view(B, S, 6, D)
        kind, w, b, eps = nrm if nrm else (0, None, None, 1e-6)
        kernels.qk_norm_rope([(want, w, kind, rp is not None, b)], eps=eps, cos=cos, sin=sin,
                             rope_seq_start=rp[0] if rp else 0, rope_row0=rp[1] if rp else 0)
        want2 = kernels.linear_fused(x2, lin2.weight, lin2.bias, **kw)
        want3 = kernels.linear_fused(x, lin.weight, lin.bias, "gelu_tanh", **kw)
    torch.cuda.synchronize()
    assert _C.device_status(0, clear=True)[0] == 0
    if tile != (0, 0, 0):  # the library may choose other tile shapes for one item than for three: another order of sums
        assert torch.equal(got.view(B, S, 6, D), want) and torch.equal(got2, want2) and torch.equal(got3, want3)
    _check(got.view(B, S, 6, D), want)
    _check(got2, want2)
    _check(got3, want3)
    assert (wide[..., :64] == 3).all()


def test_linear_group_argument_errors():
    from hetu_dit_b200 import _C, kernels
    lin, x, nrm, _ = _group_case(128, 1, None, 40, 2, torch.bfloat16, 1)
    cos = torch.zeros(30, 128, device=DEV)
    with torch.no_grad():
        for it in (kernels.Lin(x, lin, "norm_rope", head_dim=96), kernels.Lin(x, lin, "norm_rope", head_dim=128, rope=(0, 0)),
                   kernels.Lin(x, lin, "norm_rope", head_dim=128, norm=(2, None, None, 1e-6)),
                   kernels.Lin(x[:, :20].contiguous(), lin, "norm_rope", head_dim=128, rope=(0, 0))):
            with pytest.raises((_C.HditError, ValueError)):
                kernels.linear_group([it], cos, cos)
        with pytest.raises(ValueError):
            kernels.linear_group([kernels.Lin(x, lin)] * 9)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_linear_group_on_row_slices_of_a_batch(dtype):
    """Rows that are a slice of every batch entry (the image and text rows of one attention output): one launch with an item
    per entry, the bits of a call on contiguous copies, nothing written outside the slices."""
    from hetu_dit_b200 import _C, kernels
    gen = torch.Generator().manual_seed(9)

    def mk(*shape):
        return torch.randn(*shape, generator=gen).to(dtype).to(DEV)

    x, gate, w = mk(2, 300, 256), mk(2, 192), (1 + 0.2 * mk(64))
    lin = torch.nn.Linear(256, 192, device=DEV, dtype=dtype)
    cos, sin = (torch.randn(300, 64, generator=gen).to(DEV) for _ in range(2))
    kw = dict(tile_m=128, tile_n=128)  # one tile shape on both sides: one order of sums
    gated, normed = (torch.full((2, 320, 208), 7.0, dtype=dtype, device=DEV) for _ in range(2))
    res = mk(2, 320, 192)
    with torch.no_grad():
        items, want = [], []
        for lo, hi, rope in ((0, 223, None), (223, 300, (13, 4))):
            xs, whole = x[:, lo:hi], x[:, lo:hi].contiguous()
            items += [kernels.Lin(xs, lin, "gate_residual", residual=res[:, 5 + lo:5 + hi], gate=gate, out=gated[:, 5 + lo:5 + hi, 8:200]),
                      kernels.Lin(xs, lin, "norm_rope", head_dim=64, norm=(1, w, None, 1e-6), rope=rope, out=normed[:, 5 + lo:5 + hi, 8:200])]
            want += kernels.linear_group([
                kernels.Lin(whole, lin, "gate_residual", residual=res[:, 5 + lo:5 + hi].contiguous(), gate=gate),
                kernels.Lin(whole, lin, "norm_rope", head_dim=64, norm=(1, w, None, 1e-6), rope=rope)], cos, sin, **kw)
            _check(want[-2], _want(whole, lin.weight, lin.bias, "gate_residual", res[:, 5 + lo:5 + hi], gate))
        before = kernels.launch_count()
        got = kernels.linear_group(items, cos, sin, **kw)
        assert kernels.launch_count() == before + 1
    assert all(torch.equal(a, b) for a, b in zip(got, want))
    for buf, own in ((gated, (want[0], want[2])), (normed, (want[1], want[3]))):
        untouched = torch.full_like(buf, 7.0)
        untouched[:, 5:305, 8:200] = torch.cat(own, dim=1)
        assert torch.equal(buf, untouched)
    assert _C.device_status(0, clear=True)[0] == 0


def _linear_kernels(call):
    """What call() returns and the names of the linear kernels that it launched."""
    from torch.profiler import ProfilerActivity, profile
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        result = call()
        torch.cuda.synchronize()
    return result, {e.name for e in prof.events() if "linear_fused_kernel" in e.name}


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("width,B,S,K,N", [(192, 1, 256, 64, 384), (192, 1, 250, 200, 376), (192, 1, 129, 1160, 328),
                                           (192, 2, 250, 3072, 1152), (128, 1, 256, 64, 256), (128, 1, 140, 200, 136),
                                           (128, 2, 120, 4160, 256)])
def test_narrow_tiles_of_a_cta_pair(width, B, S, K, N, dtype):
    """Sizes for which a launch on four SMs takes 256 x 192 or 256 x 128 tiles of a CTA pair: every tail, ragged rows and
    columns, and (more tiles than pairs) both accumulators in turn. The order of sums is that of 256 x 256 tiles, so the
    bits are too."""
    from hetu_dit_b200 import _C, kernels
    x, w, b, res, gate = _inputs(B, S, K, N, dtype, K + N)
    got, names = _linear_kernels(lambda: {
        ep: kernels.linear_fused(x, w, b, epilogue=ep, residual=res, gate=gate, max_ctas=4)
        for ep in ("bias", "gelu_tanh", "gate_residual")})
    assert names and all(f"<128, {width}, true" in n for n in names), names
    for ep, y in got.items():
        _check(y, _want(x, w, b, ep, res, gate))
        assert torch.equal(y, kernels.linear_fused(x, w, b, epilogue=ep, residual=res, gate=gate, cta_pair=2))
    torch.cuda.synchronize()
    assert _C.device_status(0, clear=True)[0] == 0


@pytest.mark.parametrize("D,norm,rope", [(64, 1, None), (64, 2, (3, 1)), (128, 1, (3, 1)), (128, 0, (0, 0))])
@pytest.mark.parametrize("S", [130, 250, 520])
def test_norm_rope_tail_on_narrow_tiles(D, norm, rope, S):
    """The norm and rotation tail where a tile is 192 columns (heads of 64) or 128 columns wide (either head size; a warp
    team may begin in the middle of a head): the bits of 256-column tiles. Each width runs for some number of SMs, by the
    kernels' names, except 128 columns at heads of 64 and three rows of tiles."""
    from hetu_dit_b200 import _C, kernels
    lin, x, nrm, rp = _group_case(D, norm, rope, S, 1, torch.bfloat16, 7 * D + S)
    gen = torch.Generator().manual_seed(4)
    cos, sin = (torch.randn(S + 8, D, generator=gen).to(DEV) for _ in range(2))
    with torch.no_grad():
        items = lambda: [kernels.Lin(x, lin, "norm_rope", head_dim=D, norm=nrm, rope=rp)]
        want, = kernels.linear_group(items(), cos, sin, cta_pair=2)
        seen = set()
        for ctas in (4, 6, 8, 12):
            (got,), names = _linear_kernels(lambda: kernels.linear_group(items(), cos, sin, max_ctas=ctas))
            assert torch.equal(got, want), ctas
            seen |= {w for w in (128, 192) if any(f"<128, {w}, true" in n for n in names)}
    assert seen == ({128} if D == 128 else {192} if S == 520 else {128, 192})
    torch.cuda.synchronize()
    assert _C.device_status(0, clear=True)[0] == 0
