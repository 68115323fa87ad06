"""Numerics of the tcgen05 GEMM family against fp32 PyTorch statements of the same ops."""
import pytest
import torch

from physicsnemo_b200 import ops
from physicsnemo_b200.ops import gemm as G

pytestmark = pytest.mark.gpu


def _rand(*shape, scale=1.0):
    return (torch.randn(*shape, device="cuda") * scale).to(torch.bfloat16)


def _close(out, ref, tol=2e-2):
    """Element-wise: |out - ref| <= tol/2 * |ref| + tol/2 * rms(ref) (bf16 rounding is 0.4 % of the element; the floor
    covers entries that are small because their terms cancel, whose error scales with the typical size instead)."""
    out, ref = out.float(), ref.float()
    rms = ref.pow(2).mean().sqrt().item() + 1e-6
    excess = (out - ref).abs() - (0.5 * tol * ref.abs() + 0.5 * tol * rms)
    worst = excess.max().item()
    assert worst <= 0, f"worst excess over the element-wise bound {worst} (rms of the reference {rms})"


@pytest.mark.parametrize("M,N,K", [(128, 128, 64), (300, 256, 256), (1000, 64, 128), (257, 264, 72), (20000, 512, 256)])
@pytest.mark.parametrize("bn", [0, 128])
def test_gemm_tn_plain(M, N, K, bn):
    a, b = _rand(M, K), _rand(N, K, scale=0.1)
    bias = torch.randn(N, device="cuda")
    out = ops.gemm_tn(a, b, bias=bias, bn=bn)
    ref, _ = ops.gemm_tn_reference(a, b, bias=bias)
    _close(out, ref)
    assert ops.device_error() == 0


@pytest.mark.parametrize("act", [G.ACT_GELU, G.ACT_SILU, G.ACT_RELU, G.ACT_SOFTMAX64])
def test_gemm_tn_activation_and_z(act):
    M, N, K = 777, 256, 128
    a, b = _rand(M, K), _rand(N, K, scale=0.2)
    bias = torch.randn(N, device="cuda")
    scale = torch.rand(N, device="cuda") + 0.5
    out, z = ops.gemm_tn(a, b, bias=bias, scale=scale, act=act, z_out=True)
    ref, zref = ops.gemm_tn_reference(a, b, bias=bias, scale=scale, act=act)
    _close(z, zref)
    _close(out, ref)
    out2 = ops.gemm_tn(a, b, bias=bias, scale=scale, act=act)
    _close(out2, ref)


@pytest.mark.parametrize("aux_mode", [G.AUX_ADD, G.AUX_DGELU, G.AUX_DSILU, G.AUX_DRELU, G.AUX_DSOFTMAX])
def test_gemm_tn_aux(aux_mode):
    M, N, K = 1500, 384, 192
    a, b = _rand(M, K), _rand(N, K, scale=0.2)
    if aux_mode == G.AUX_DSOFTMAX:
        aux = torch.softmax(torch.randn(M, N // 64, 64, device="cuda"), -1).reshape(M, N).to(torch.bfloat16)
    else:
        aux = _rand(M, N)
    scale = torch.rand(N, device="cuda") + 0.5
    grp = torch.zeros(N // 64, device="cuda") if aux_mode == G.AUX_DSOFTMAX else None
    out = ops.gemm_tn(a, b, aux=aux, aux_mode=aux_mode, scale=scale, scale_post=True, group_out=grp)
    ref, _ = ops.gemm_tn_reference(a, b, aux=aux, aux_mode=aux_mode, scale=scale, scale_post=True)
    _close(out, ref, tol=3e-2)
    if grp is not None:
        y = (a.float() @ b.float().t()).reshape(M, -1, 64)
        p = aux.float().reshape(M, -1, 64)
        ds = p * (y - (y * p).sum(-1, keepdim=True))
        gref = (ds * torch.log(p.clamp_min(1e-30)) * (p > 0)).sum((0, 2))
        _close(grp, gref, tol=5e-2)
    assert ops.device_error() == 0


def test_gemm_tn_k_concat():
    M, N, K1, K2 = 900, 256, 128, 192
    a, a2, b = _rand(M, K1), _rand(M, K2), _rand(N, K1 + K2, scale=0.1)
    out = ops.gemm_tn(a, b, a2=a2)
    ref, _ = ops.gemm_tn_reference(a, b, a2=a2)
    _close(out, ref)


@pytest.mark.parametrize("M,Na,Nb", [(64, 128, 128), (5000, 256, 256), (4097, 512, 256), (1000, 64, 32), (30000, 1024, 256),
                                     # >= 8192 rows and >= 256 output rows: the CTA-pair kernel (ragged edges in all three sizes)
                                     (32400, 768, 3072), (9001, 264, 136), (8192, 256, 128)])
def test_gemm_nt(M, Na, Nb):
    a, b = _rand(M, Na, scale=0.3), _rand(M, Nb, scale=0.3)
    out, cs = ops.gemm_nt(a, b, colsum=True)
    ref = a.float().t() @ b.float()
    _close(out, ref, tol=1e-2)
    _close(cs, a.float().sum(0), tol=1e-2)
    assert ops.device_error() == 0


def test_gradients_of_a_weight_and_its_bias_are_two_buffers():
    """A bias' gradient that is held or saved holds no weight's, and neither notices what is done to the other in place."""
    x = torch.randn(300, 128, device="cuda").bfloat16()
    params = [torch.randn(256, 128, device="cuda", requires_grad=True), torch.randn(256, device="cuda", requires_grad=True)]
    ops.mlp_chain(x, params[:1], params[1:], [G.ACT_NONE]).float().sum().backward()
    for p in params:
        assert p.grad.untyped_storage().nbytes() == p.grad.nbytes
    dw, db = ops.gemm_nt(x, x, colsum=True)
    before = dw._version
    db.add_(1)
    assert dw._version == before and dw.untyped_storage().data_ptr() != db.untyped_storage().data_ptr()


@pytest.mark.parametrize("P,Mp,N,K", [(8, 8320, 192, 192), (3, 256, 64, 64), (2, 384, 264, 136)])
def test_gemm_stacked_batches(P, Mp, N, K):
    """`P` equal problems in one launch: forward with bias + ReLU, data gradient with the ReLU mask, weight gradient
    with column sums — each against the per-problem fp32 statement."""
    a, w = _rand(P, Mp, K), _rand(P, N, K, scale=0.1)
    bias = torch.randn(P, N, device="cuda")
    out = G.gemm_tn_stacked(a, w, bias=bias, act=G.ACT_RELU)
    ref = torch.relu(torch.einsum("pmk,pnk->pmn", a.float(), w.float()) + bias[:, None])
    _close(out, ref)
    gy = _rand(P, Mp, N)
    wt = w.transpose(1, 2).contiguous()
    # the mask has the product's shape: dx = (gy @ w) where aux > 0
    dref = torch.einsum("pmn,pnk->pmk", gy.float(), w.float())
    aux = _rand(P, Mp, K)
    dx = G.gemm_tn_stacked(gy, wt, aux=aux, aux_mode=G.AUX_DRELU)
    _close(dx, dref * (aux.float() > 0))
    dw = torch.zeros(P, N, K, device="cuda")
    db = torch.zeros(P, N, device="cuda")
    G.gemm_nt_stacked(gy, a, dw, db)
    _close(dw, torch.einsum("pmn,pmk->pnk", gy.float(), a.float()), tol=1e-2)
    _close(db, gy.float().sum(1), tol=1e-2)
    assert ops.device_error() == 0


@pytest.mark.parametrize("C", [128, 256, 768])
def test_layernorm(C):
    M = 3001
    x = _rand(M, C).requires_grad_(True)
    w = (torch.rand(C, device="cuda") + 0.5).requires_grad_(True)
    b = torch.randn(C, device="cuda").requires_grad_(True)
    y = ops.layer_norm(x, w, b)
    dy = _rand(M, C)
    y.backward(dy)
    xr = x.detach().float().requires_grad_(True)
    wr, br = w.detach().clone().requires_grad_(True), b.detach().clone().requires_grad_(True)
    yr = torch.nn.functional.layer_norm(xr, (C,), wr, br)
    yr.backward(dy.float())
    _close(y, yr)
    _close(x.grad, xr.grad, tol=3e-2)
    _close(w.grad, wr.grad, tol=2e-2)
    _close(b.grad, br.grad, tol=2e-2)


def _layernorm_against_64_bits(M, C, post=False, residual=False):
    """One forward and backward; bf16 results carry one rounding (2^-9 at most, 1.7e-3 in the 2-norm), the column sums are fp32."""
    x, r, dy, dr = (_rand(M, C) for _ in range(4))
    w, b = torch.rand(C, device="cuda") + 0.5, torch.randn(C, device="cuda")
    got = [t.clone().requires_grad_(True) for t in (x, r, w, b)]
    ref = [t.double().requires_grad_(True) for t in (x, r, w, b)]
    y = ops.layer_norm(got[0], got[2], got[3], post=got[1] if post else None, return_residual=residual)
    yr = torch.nn.functional.layer_norm(ref[0], (C,), ref[2], ref[3]) + (ref[1] if post else 0)
    if residual:
        y, alias = y
        torch.autograd.backward([y, alias], [dy, dr])
        torch.autograd.backward([yr, ref[0] * 1], [dy.double(), dr.double()])
    else:
        y.backward(dy)
        yr.backward(dy.double())
    rel = lambda a, e: float((a.double() - e).norm() / e.norm())  # noqa: E731
    assert rel(y.detach(), yr.detach()) < 4e-3 and rel(got[0].grad, ref[0].grad) < 4e-3
    assert rel(got[2].grad, ref[2].grad) < 2e-5 and rel(got[3].grad, ref[3].grad) < 2e-5
    if post:
        assert torch.equal(got[1].grad, dy)


@pytest.mark.parametrize("M", [1, 1531, 60001])
@pytest.mark.parametrize("C", [8, 16, 24, 32, 40])
def test_layernorm_narrow_rows(M, C):
    """Rows so short that the fold of the column sums is larger than the ring of row tiles."""
    for _ in range(5):
        _layernorm_against_64_bits(M, C)
    assert ops.device_error() == 0


def test_mlp_chain_matches_torch():
    M = 2050
    x = _rand(M, 6).requires_grad_(True)
    res = _rand(M, 256).requires_grad_(True)
    ws = [torch.randn(512, 6, device="cuda") * 0.3, torch.randn(256, 512, device="cuda") * 0.05]
    bs = [torch.randn(512, device="cuda") * 0.1, torch.randn(256, device="cuda") * 0.1]
    for t in ws + bs:
        t.requires_grad_(True)
    y = ops.mlp_chain(x, ws, bs, [G.ACT_GELU, G.ACT_NONE], residual=res)
    dy = _rand(M, 256)
    y.backward(dy)
    got = [x.grad, res.grad] + [t.grad for t in ws + bs]
    xr = x.detach().float().requires_grad_(True)
    rr = res.detach().float().requires_grad_(True)
    wr = [t.detach().clone().requires_grad_(True) for t in ws]
    br = [t.detach().clone().requires_grad_(True) for t in bs]
    h = torch.nn.functional.gelu(xr @ wr[0].t() + br[0]) @ wr[1].t() + br[1] + rr
    h.backward(dy.float())
    _close(y, h, tol=3e-2)
    for g, r in zip(got, [xr.grad, rr.grad] + [t.grad for t in wr + br]):
        _close(g, r, tol=4e-2)
    assert ops.device_error() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("M,N,K", [(1000, 128, 128), (257, 72, 72), (90000, 128, 320), (512, 128, 64)])
def test_gemm_tn_split_m_tiles(M, N, K):
    """256-row x 128-column tiles (two row sub-tiles sharing one B tile), forced with bn = -256 and, for the large M,
    chosen by the launcher itself."""
    a, b = _rand(M, K), _rand(N, K, scale=0.1)
    bias = torch.randn(N, device="cuda")
    ref, _ = ops.gemm_tn_reference(a, b, bias=bias, act=G.ACT_SILU)
    _close(ops.gemm_tn(a, b, bias=bias, act=G.ACT_SILU, bn=-256), ref)
    _close(ops.gemm_tn(a, b, bias=bias, act=G.ACT_SILU), ref)
    assert ops.device_error() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(2, 64, 128, 24, 40, 3), (1, 128, 64, 17, 33, 3), (3, 64, 72, 8, 16, 1), (1, 192, 256, 40, 24, 5),
                                   (1, 128, 128, 296, 272, 3), (1, 64, 96, 320, 256, 1),
                                   # >= 8192 pixels and K >= 512: the CTA-pair tiles (256 x 128 and 256 x 256), with ragged image
                                   # edges, a ragged channel edge, an odd number of pixel tiles and a 1 x 1 window
                                   (1, 128, 256, 90, 100, 3), (1, 64, 192, 100, 90, 3), (1, 128, 128, 72, 144, 3),
                                   (1, 512, 128, 96, 96, 1), (1, 256, 256, 64, 136, 3)])
def test_conv2d_same_implicit_gemm(shape):
    from physicsnemo_b200.ops import conv as C

    n, cin, cout, h, w, k = shape
    torch.manual_seed(0)
    x = torch.randn(n, cin, h, w, device="cuda").to(memory_format=torch.channels_last).requires_grad_(True)
    wt = (torch.randn(cout, cin, k, k, device="cuda") / (cin * k * k) ** 0.5).requires_grad_(True)
    b = torch.randn(cout, device="cuda").requires_grad_(True)
    assert C.supported(x, wt)
    y = C.conv2d_same(x, wt, b)
    assert y.shape == (n, cout, h, w) and y.is_contiguous(memory_format=torch.channels_last)
    xr, wr, br = (t.detach().clone().requires_grad_(True) for t in (x, wt, b))
    ref = torch.nn.functional.conv2d(xr, wr, br, padding=k // 2)
    assert (y.float() - ref).abs().max() < 4e-2
    dy = torch.randn_like(ref)
    y.backward(dy.to(y.dtype))
    ref.backward(dy)
    assert (x.grad - xr.grad).abs().max() < 6e-2 * max(1.0, float(xr.grad.abs().max()))
    assert (wt.grad - wr.grad).abs().max() < 3e-2 * float(wr.grad.abs().max())
    assert (b.grad - br.grad).abs().max() < 2e-2 * float(br.grad.abs().max())
    fused = C.conv2d_same(x.detach(), wt.detach(), b.detach(), act="silu")
    assert (fused.float() - torch.nn.functional.silu(ref.detach())).abs().max() < 4e-2


@pytest.mark.gpu
@pytest.mark.parametrize("n,h,w,cin,cout", [(1, 1, 1, 64, 64), (1, 8, 16, 64, 72), (3, 7, 15, 128, 128), (1, 17, 33, 192, 136), (2, 41, 50, 64, 256),
                                            (1, 64, 64, 512, 512), (1, 130, 126, 128, 384), (1, 200, 176, 128, 256)])
def test_conv3x3_forward_by_columns_of_taps(n, h, w, cin, cout):
    """One tile and less, an odd number of pixel tiles (half a pair is empty), ragged edges and channels, narrow and wide tiles.  Against
    64 bits on the same bf16 operands only the rounding of the result is left: at most 2^-8 of a value."""
    from physicsnemo_b200.ops import conv as C

    g = torch.Generator(device="cuda").manual_seed(n * h + w)
    x = torch.randn(n, cin, h, w, generator=g, device="cuda").bfloat16().contiguous(memory_format=torch.channels_last)
    wt = (torch.randn(cout, cin, 3, 3, generator=g, device="cuda") / (9 * cin) ** 0.5).bfloat16()
    b = torch.randn(cout, generator=g, device="cuda")
    y = C.conv2d_same(x, wt, b)
    ref = torch.nn.functional.conv2d(x.double(), wt.double(), b.double(), padding=1)
    assert float(((y - ref).abs() - 2.0 ** -8 * ref.abs()).max()) < 1e-4            # sums that cancel: 4 608 terms of fp32 rounding
    assert ops.device_error() == 0


@pytest.mark.parametrize("n,h,w,cin,cout", [(1, 1, 1, 64, 64), (3, 7, 15, 128, 128), (1, 17, 33, 192, 136), (2, 41, 50, 64, 264), (1, 64, 64, 512, 512),
                                            (1, 130, 126, 128, 384)])
def test_conv3x3_tiles_of_both_widths(n, h, w, cin, cout):
    """Every shape on tiles of 128 and of 256 output channels, whichever the rule would take; a tile that does not apply is refused."""
    import ctypes as c

    from physicsnemo_b200.ops import _lib
    from physicsnemo_b200.ops import conv as C

    conv = _lib.load(required=True)["pnm_conv2d_nhwc"]
    conv.argtypes, conv.restype = [c.c_void_p] * 3 + [c.c_int] * 6 + [c.c_void_p] + [c.c_int] * 3 + [c.c_void_p], c.c_int
    g = torch.Generator(device="cuda").manual_seed(n * h + w)
    x = torch.randn(n, h, w, cin, generator=g, device="cuda").bfloat16()
    wt = (torch.randn(cout, cin, 3, 3, generator=g, device="cuda") / (9 * cin) ** 0.5).bfloat16()
    b = torch.randn(cout, generator=g, device="cuda")
    packed = C._forward_operand(wt, cin, cout)
    ref = torch.nn.functional.conv2d(x.double().permute(0, 3, 1, 2), wt.double(), b.double(), padding=1).permute(0, 2, 3, 1)
    for bn in (1128, 1256):
        y = torch.full((n, h, w, cout), float("nan"), device="cuda", dtype=torch.bfloat16)

        def call(ksize, max_ctas):
            return conv(x.data_ptr(), packed.data_ptr(), y.data_ptr(), n, h, w, cin, cout, ksize, b.data_ptr(), 0, bn, max_ctas, _lib.stream())

        assert call(3, 0) == 0
        assert float(((y - ref).abs() - 2.0 ** -8 * ref.abs()).max()) < 1e-4        # as above
        assert call(1, 0) == call(3, 4) == -2
    assert ops.device_error() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("n,h,w,cin,cout", [(1, 4, 16, 128, 128), (2, 33, 31, 64, 64), (1, 45, 50, 192, 72), (3, 29, 47, 128, 200),
                                            (1, 64, 64, 320, 136), (1, 130, 126, 128, 256), (2, 24, 24, 512, 512)])
def test_conv3x3_weight_gradient_by_columns_of_taps(n, h, w, cin, cout):
    """Patches that the image's edges cut, one or two boxes of 64 input channels, ragged output channels; (1, 4, 16) is left to the
    reduction GEMM.  A product of two bf16 values is exact in fp32 and 16 of them enter an accumulator together: each of the
    pixels / 16 additions may lose 2^-23 of the sum."""
    from physicsnemo_b200.ops import conv as C

    g = torch.Generator(device="cuda").manual_seed(n * h + w)
    x = torch.randn(n, h, w, cin, generator=g, device="cuda").bfloat16()
    dy = torch.randn(n, h, w, cout, generator=g, device="cuda").bfloat16()
    dw, db = C.wgrad3x3(dy, x, True)
    ref = torch.nn.grad.conv2d_weight(x.permute(0, 3, 1, 2).double(), (cout, cin, 3, 3), dy.permute(0, 3, 1, 2).double(), padding=1)
    ref, ref_b = ref.permute(0, 2, 3, 1).reshape(cout, -1), dy.double().sum((0, 1, 2))
    bound = max(16, n * h * w / 16) * 2.0 ** -23
    assert float((dw - ref).norm() / ref.norm()) < bound
    assert float((db - ref_b).norm() / ref_b.norm()) < bound
    assert ops.device_error() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("M,N,K", [(2048, 1024, 256), (2999, 1096, 264), (2304, 1032, 504), (2100, 1024, 512)])
def test_gemm_tn_two_outputs_of_short_products(M, N, K):
    """Two outputs on CTA pairs, two pairs of staging buffers at K = 256 and one above: ragged edges, several blocks per warp."""
    a, b, bias = _rand(M, K), _rand(N, K, scale=K ** -0.5), torch.randn(N, device="cuda")
    y, z = G.gemm_tn(a, b, bias=bias, act=G.ACT_GELU, z_out=True)
    zr = a.double() @ b.double().t() + bias.double()
    assert float(((z - zr).abs() - 2.0 ** -8 * zr.abs()).max()) < 1e-4            # rounded once
    # the kernels' GELU is the tanh form: within 1e-3 of the erf form
    yr = torch.nn.functional.gelu(zr, approximate="tanh")
    assert float(((y - yr).abs() - 2.0 ** -8 * yr.abs()).max()) < 2e-3
    assert ops.device_error() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("skip", [1, 2, 3])
@pytest.mark.parametrize("M,N,K", [(300, 128, 72), (300, 320, 64), (90000, 128, 64), (40000, 256, 128), (2048, 1024, 256), (2304, 576, 512)])
def test_vectors_that_start_off_a_16_byte_boundary(M, N, K, skip):
    """Bias and scale as slices of a flat buffer, `skip` elements from its start, on every kind of tile and with every kind of epilogue, and
    in a convolution: what an aligned copy gives, bit for bit."""
    from physicsnemo_b200.ops import conv as C

    a, b, aux = _rand(M, K), _rand(N, K, scale=K ** -0.5), _rand(M, N)
    flat = torch.randn(2 * N + 8, device="cuda")
    bias, scale = flat[skip:skip + N], flat[N + 4 + skip:2 * N + 4 + skip]
    assert bias.data_ptr() % 16 == scale.data_ptr() % 16 == 4 * skip
    forms = [dict(bias=bias), dict(bias=bias, act=G.ACT_GELU), dict(bias=bias, scale=scale), dict(bias=bias, scale=scale, scale_post=True),
             dict(bias=bias, act=G.ACT_SILU, z_out=True), dict(bias=bias, aux=aux, aux_mode=G.AUX_ADD), dict(bias=bias, aux=aux, aux_mode=G.AUX_DGELU)]
    if N % 64 == 0:
        forms += [dict(bias=bias, scale=scale, act=G.ACT_SOFTMAX64), dict(bias=bias, scale=scale, scale_post=True, aux=aux, aux_mode=G.AUX_DSOFTMAX)]
    for form in forms:
        own = {k: v.clone() if k in ("bias", "scale") else v for k, v in form.items()}
        out, want = G.gemm_tn(a, b, **form), G.gemm_tn(a, b, **own)
        for u, v in zip(*((t if isinstance(t, tuple) else (t,)) for t in (out, want))):
            assert torch.equal(u, v)
    x = _rand(1, 64, 24, 40).contiguous(memory_format=torch.channels_last)
    for k in (1, 3):
        w = _rand(N, 64, k, k, scale=0.05)
        assert torch.equal(C.conv2d_same(x, w, bias), C.conv2d_same(x, w, bias.clone()))
    assert ops.device_error() == 0


@pytest.mark.parametrize("M,N,K", [(2048, 256, 512), (4000, 768, 1024), (32400, 1096, 768), (2304, 520, 584)])
@pytest.mark.parametrize("mode", ["plain", "gelu_z", "add", "dgelu", "drelu"])
def test_gemm_tn_cta_pair_tiles(M, N, K, mode):
    """Compute-bound shapes (K >= 512, N >= 256, M >= 2048) run as 256 x 256 tiles on CTA pairs (cta_group::2): ragged M,
    N and K edges, every epilogue the pair kernel carries, against the fp32 statement and against the single-CTA kernel."""
    a, b = _rand(M, K), _rand(N, K, scale=0.05)
    bias = torch.randn(N, device="cuda")
    aux = _rand(M, N)
    kw = {"plain": dict(bias=bias), "gelu_z": dict(bias=bias, act=G.ACT_GELU, z_out=True),
          "add": dict(bias=bias, aux=aux, aux_mode=G.AUX_ADD), "dgelu": dict(aux=aux, aux_mode=G.AUX_DGELU),
          "drelu": dict(aux=aux, aux_mode=G.AUX_DRELU)}[mode]
    out = ops.gemm_tn(a, b, **kw)
    ref_kw = {k: v for k, v in kw.items() if k != "z_out"}
    ref, zref = ops.gemm_tn_reference(a, b, **ref_kw)
    single = ops.gemm_tn(a, b, bn=128 if mode == "plain" else 0, max_ctas=148, **kw)      # max_ctas keeps it off the pair kernel
    if mode == "gelu_z":
        (out, z), (single, zs) = out, single
        _close(z, zref)
        _close(z, zs, tol=1e-2)
    _close(out, ref)
    assert (out.float() - single.float()).abs().max().item() <= 2e-2 * ref.abs().max().item()
    assert ops.device_error() == 0


def test_weight_copy_of_another_stream_is_not_used_before_it_is_made():
    w = torch.nn.Parameter(torch.randn(256, 128, device="cuda"))
    ref = w.detach().bfloat16()
    busy, other = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(busy):
        torch.cuda._sleep(100_000_000)                   # about 50 ms: the conversion below waits behind it
        first = G._bf16_weight(w)
    with torch.cuda.stream(other):
        got = G._bf16_weight(w).clone()
        other.synchronize()
        assert torch.equal(got, ref) and G._bf16_weight(w) is not first
    with torch.cuda.stream(busy):
        assert G._bf16_weight(w) is first
    torch.cuda.synchronize()
    assert torch.equal(first, ref)


@pytest.mark.parametrize("N", [256, 384, 448, 1000, 136])
@pytest.mark.parametrize("aux_mode", [G.AUX_DGELU, G.AUX_DSILU, G.AUX_DSOFTMAX])
@pytest.mark.parametrize("form", ["plain", "bias, scale before", "bias, scale after", "two sources, activation"])
def test_gemm_tn_wide_aux_tiles(aux_mode, N, form):
    """256-column tiles with an auxiliary operand need a tile per SM (157 row tiles here): ragged rows, a last tile of 128, 192, 232 or
    136 columns, and all that the epilogue does before and after the operand."""
    if aux_mode == G.AUX_DSOFTMAX:
        N = N // 64 * 64
    M, K1, K2 = 20001, 128, 64
    a, a2, b = _rand(M, K1), _rand(M, K2), _rand(N, K1 + K2, scale=0.2)
    aux = torch.softmax(torch.randn(M, N // 64, 64, device="cuda"), -1).reshape(M, N).bfloat16() if aux_mode == G.AUX_DSOFTMAX else _rand(M, N)
    kw = {"aux": aux, "aux_mode": aux_mode}
    if form == "two sources, activation":
        kw |= {"a2": a2, "act": G.ACT_SILU}
    else:
        a = torch.cat([a, a2], 1)
        kw["scale_post"] = form != "bias, scale before"
        if form != "plain":
            kw |= {"bias": torch.randn(N, device="cuda"), "scale": torch.rand(N, device="cuda") + 0.5}
        else:
            kw["scale"] = torch.ones(N, device="cuda")           # keeps the deep shapes off the CTA-pair kernel
    grp = torch.zeros(N // 64, device="cuda") if aux_mode == G.AUX_DSOFTMAX and form == "bias, scale after" else None
    out = ops.gemm_tn(a, b, group_out=grp, **kw)
    ref, z = ops.gemm_tn_reference(a, b, **kw)
    _close(out, ref, tol=3e-2)
    if grp is not None:
        y, p = z.reshape(M, -1, 64), aux.float().reshape(M, -1, 64)
        ds = p * (y - (y * p).sum(-1, keepdim=True))
        _close(grp, (ds * torch.log(p.clamp_min(1e-30)) * (p > 0)).double().sum((0, 2)), tol=5e-2)
    assert ops.device_error() == 0


@pytest.mark.parametrize("form", [{}, {"post": True}, {"residual": True}, {"post": True, "residual": True}])
@pytest.mark.parametrize("C", [8, 128, 200, 256, 512, 768, 1024])
def test_layernorm_rings_that_wrap(C, form):
    """Rows enough that every CTA uses every stage of its ring again, with a last tile that is not full."""
    _layernorm_against_64_bits(120001 if C <= 256 else 60001, C, **form)
    assert ops.device_error() == 0
