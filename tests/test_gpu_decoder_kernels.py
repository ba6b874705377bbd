"""Residual add + RMSNorm, rotary embedding and SwiGLU kernels against plain PyTorch."""
import pytest
import torch
import torch.nn.functional as F

from flashoverlap_b200 import ops
from flashoverlap_b200.models.decoder_layer import _rope
from flashoverlap_b200.utils import layout

pytestmark = pytest.mark.gpu
DTYPES = [torch.bfloat16, torch.float16]
ULP = {torch.bfloat16: 2.0 ** -7, torch.float16: 2.0 ** -10}     # largest spacing of neighbours over the value


def _op():
    return torch.ops.flashoverlap_op


# one vector, a remainder in every vectors-per-thread variant, the largest row; one row, several rows per CTA
@pytest.mark.parametrize("dt", DTYPES)
@pytest.mark.parametrize("rows,dim", [(1, 8), (3, 2040), (130, 2056), (1500, 4104), (5000, 1024), (33, 8200), (9, 16384)])
def test_add_rmsnorm(cuda, dt, rows, dim):
    x, t = torch.randn(rows, dim, device=cuda).to(dt), torch.randn(rows, dim, device=cuda).to(dt)
    w = (1 + 0.02 * torch.randn(dim, device=cuda)).to(dt)
    h, y = torch.empty_like(x), torch.empty_like(x)
    _op().add_rmsnorm(x, t, h, y, w, 1e-5)
    assert torch.equal(h, x + t)
    assert torch.equal(y, ops.rmsnorm(h, w, 1e-5))
    in_place, y2 = x.clone(), torch.empty_like(x)
    _op().add_rmsnorm(in_place, t, in_place, y2, w, 1e-5)
    assert torch.equal(in_place, h) and torch.equal(y2, y)
    ref = layout.rmsnorm_ref(x + t, w, 1e-5).double()
    assert ((y.double() - ref).abs() <= 2 * ULP[dt] * ref.abs() + 1e-6).all()     # the norm rounds twice


def test_add_rmsnorm_refuses(cuda):
    x = torch.zeros(4, 64, device=cuda, dtype=torch.bfloat16)
    w = torch.ones(64, device=cuda, dtype=torch.bfloat16)
    for bad in (x[:, :32], x.half(), x[:2], x.cpu()):
        with pytest.raises(RuntimeError):
            _op().add_rmsnorm(x, bad, x.clone(), x.clone(), w, 1e-5)


@pytest.mark.parametrize("dt", DTYPES)
@pytest.mark.parametrize("B,S,heads,extra,hd", [(1, 128, 9, 1, 128), (2, 96, 1, 0, 64), (3, 33, 17, 2, 8), (1, 5000, 8, 8, 128)])
def test_rope(cuda, dt, B, S, heads, extra, hd):
    qkv = torch.randn(B * S, (heads + extra) * hd, device=cuda).to(dt)
    out = qkv.clone()
    _op().rope_(out, S, heads, hd, 500000.0)
    got = out[:, :heads * hd].view(B, S, heads, hd).transpose(1, 2)
    x = qkv[:, :heads * hd].view(B, S, heads, hd).transpose(1, 2)
    ref = _rope(x, 500000.0)
    # same angles; a pair's two products may be contracted into one rounding less, so results differ by one
    # rounding of the result or, where the products cancel, by fp32 roundings of the products
    mag = x.float().reshape(B, heads, S, hd // 2, 2).norm(dim=-1, keepdim=True).expand(-1, -1, -1, -1, 2).reshape(ref.shape)
    assert ((got.float() - ref.float()).abs() <= ULP[dt] * ref.float().abs() + 2.0 ** -20 * mag + 2.0 ** -24).all()
    assert torch.equal(out[:, heads * hd:], qkv[:, heads * hd:])


@pytest.mark.parametrize("dt", DTYPES)
@pytest.mark.parametrize("rows,f", [(1, 8), (7, 2048), (300, 2056), (64, 4104), (5000, 3584)])
def test_swiglu(cuda, dt, rows, f):
    gu = (3 * torch.randn(rows, 2 * f, device=cuda)).to(dt)
    gu[0, 0], gu[0, 1] = -60000.0, float("inf")
    y = torch.empty(rows, f, device=cuda, dtype=dt)
    _op().swiglu(gu, y)
    ref = F.silu(gu[:, :f]) * gu[:, f:]
    # silu's last fp32 bit may round the 16-bit value the other way, and the product rounds once more
    same = (y == ref) | ((y - ref).abs() <= 2 * ULP[dt] * ref.abs() + 2.0 ** -19) | (y.isnan() & ref.isnan())
    assert same.all()


@pytest.fixture(scope="module")
def impl(cuda):
    i = ops.OverlapImpl()
    i.nccl_init(0, 1, [0] * 16)
    i.cutlass_init()
    return i


# a split over K, one wave of pairs, an odd number of row tiles, N that only 128-wide tiles divide, 512-row units,
# a last wave of half-width tiles
@pytest.mark.parametrize("dt", DTYPES)
@pytest.mark.parametrize("M,N,K,algo", [(128, 1024, 512, 0), (256, 2048, 1000, 1), (640, 5376, 264, 0), (384, 1152, 128, 2),
                                        (1024, 8192, 192, 3), (1280, 4352, 264, 1)])
def test_gemm_add(cuda, impl, dt, M, N, K, algo):
    a, b = torch.randn(M, K, device=cuda).to(dt), (0.1 * torch.randn(N, K, device=cuda)).to(dt)
    r = torch.randn(M, N, device=cuda).to(dt)
    for tma, exact in ((-1, 0), (0, 0), (-1, 1)):
        impl.set_option("tma_out", tma)
        impl.set_option("exact_algo", exact)
        plain, out = torch.empty_like(r), torch.empty_like(r)
        impl.cutlass_gemm(a, b, plain, algo)
        impl.gemm_add(a, b, r, out, algo)
        assert torch.equal(out, r + plain)
        in_place = r.clone()
        impl.gemm_add(a, b, in_place, in_place, algo)
        assert torch.equal(in_place, out)
    impl.set_option("tma_out", -1)
    impl.set_option("exact_algo", 0)
    impl.check_status()


@pytest.mark.parametrize("dt", DTYPES)
@pytest.mark.parametrize("M,F_,K", [(128, 128, 64), (256, 1152, 1000), (640, 3584, 264), (4096, 2048, 512),
                                    (1280, 2176, 192), (2560, 4096, 72)])
def test_gemm_swiglu(cuda, impl, dt, M, F_, K):
    a, w = torch.randn(M, K, device=cuda).to(dt), (0.1 * torch.randn(2 * F_, K, device=cuda)).to(dt)
    out = torch.full((M, F_), float("nan"), device=cuda, dtype=dt)
    impl.gemm_swiglu(a, w, out)
    impl.check_status()
    gu = a.double() @ w.double().t()
    g, u = gu[:, :F_], gu[:, F_:]
    ref = F.silu(g) * u
    # fp32 sums: relative 2^-18 of the magnitudes that were added; silu's slope is below 1.1
    mag = a.double().abs() @ w.double().abs().t()
    bound = 0.51 * ULP[dt] * ref.abs() + 2.0 ** -18 * (1.1 * mag[:, :F_] * u.abs() + F.silu(g).abs() * mag[:, F_:]) + 2.0 ** -24
    assert ((out.double() - ref).abs() <= bound).all()


def test_one_rank_layer_copies_after_a_call(cuda):
    """The GEMM object that a one-rank layer makes for itself stays out of its copies."""
    import copy
    from flashoverlap_b200.models import DecoderConfig, TPDecoderLayer
    cfg = DecoderConfig(hidden=2048, ffn=1024, n_heads=4, n_kv_heads=2)
    layer = TPDecoderLayer(cfg, 0, 1, 1, 2048, impl="fused", device=cuda)
    x = torch.randn(2048, 2048, device=cuda).to(torch.bfloat16)
    with torch.no_grad():
        y = layer(x)
        assert torch.equal(copy.deepcopy(layer)(x), y)
    for p in layer.parameters():                       # with a graph to record: the operators that have gradients
        p.grad = None
    z = layer(x)
    z.float().sum().backward()
    assert layer.wd.grad is not None and (z - y).abs().max() <= 0.02 * y.abs().max()
    layer.check_status()


# the residual is the projection's input (h += h W^T), a part of it, and the weights' memory
@pytest.mark.parametrize("dt", DTYPES)
@pytest.mark.parametrize("where", ["A", "A shifted", "B"])
def test_add_norm_with_residual_over_an_operand(cuda, impl, dt, where):
    M, N = 2048, 2048
    mem = torch.randn(M + 128, N, device=cuda).to(dt)
    other = (0.1 * torch.randn(M, N, device=cuda)).to(dt)
    r = mem[64:64 + M] if where == "A shifted" else mem[:M]
    a, b = (other, mem[:M]) if where == "B" else (mem[:M], other)
    w, y = torch.ones(N, device=cuda, dtype=dt), torch.empty(M, N, device=cuda, dtype=dt)
    product = torch.empty_like(y)
    impl.cutlass_gemm(a, b, product, 1)
    h = r + product
    impl.gemm_reducescatter_add_rmsnorm_fused(a, b, r, y, w, 1e-5, 1)
    impl.check_status()
    assert torch.equal(r, h) and torch.equal(y, ops.rmsnorm(h, w, 1e-5))


def test_epilogue_gemms_refuse_overlapping_outputs(cuda, impl):
    mem = torch.zeros(1024 * 256, device=cuda, dtype=torch.bfloat16)
    at = lambda row: mem[row * 256:(row + 256) * 256].view(256, 256)
    a, b, r, c = at(0), at(256), at(512), at(768)
    impl.gemm_add(a, b, r, c, 0)
    for bad in (at(0), at(128), at(384), at(448), at(640)):
        with pytest.raises(RuntimeError):
            impl.gemm_add(a, b, r, bad, 0)
    half = lambda row: mem[row * 256:(row + 128) * 256].view(256, 128)
    impl.gemm_swiglu(a, b, half(512))
    for bad in (half(0), half(128), half(256), half(448)):
        with pytest.raises(RuntimeError):
            impl.gemm_swiglu(a, b, bad)
    impl.check_status()


def _one_rank_layer(cuda, T=2048):
    from flashoverlap_b200.models import DecoderConfig, TPDecoderLayer
    cfg = DecoderConfig(hidden=2048, ffn=1024, n_heads=4, n_kv_heads=2)
    return TPDecoderLayer(cfg, 0, 1, 1, T, impl="fused", device=cuda), torch.randn(T, 2048, device=cuda).to(torch.bfloat16)


def test_one_rank_layer_makes_its_gemm_object_with_itself(cuda):
    """No set-up is left for the first forward, and a capture of that first forward holds no set-up either."""
    layer, x = _one_rank_layer(cuda)
    device, made = layer._one_rank
    with torch.no_grad():
        layer.check_status()
        g = torch.cuda.CUDAGraph()
        torch.cuda.synchronize()
        with torch.cuda.graph(g):
            y = layer(x)
        layer.check_status()                       # the words are not the graph's: valid before any replay
        g.replay()
        assert torch.equal(y, layer(x))
    assert layer._one_rank[1] is made and device == x.device
    layer.check_status()


def test_one_rank_layer_copy_first_called_under_capture(cuda):
    """A copy has no object yet and makes none while a stream is captured: the operators of torch serve."""
    import copy
    layer, x = _one_rank_layer(cuda)
    twin = copy.deepcopy(layer)
    with torch.no_grad():
        ref = layer(x)
        F.scaled_dot_product_attention(*[torch.zeros(1, 4, 64, 128, device=cuda, dtype=x.dtype)] * 3, is_causal=True)
        torch.matmul(x, twin.wqkv.t())             # the library's own workspaces, ahead of the capture
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            y = twin(x)
        assert twin._one_rank is None
        twin.check_status()
        g.replay()
    # the two ways round at different places: 2 units of bf16 in the largest element
    assert (y - ref).abs().max() <= 2.0 ** -6 * ref.abs().max()
    with torch.no_grad():
        assert torch.equal(twin(x), ref) and twin._one_rank is not None
    twin.check_status()


def test_layer_check_status_reports_a_wait_that_gave_up(cuda):
    layer, x = _one_rank_layer(cuda, 128)
    own = layer._one_rank[1]
    own.set_option("timeout_ms", 50)
    own.wait_flag(1, torch.zeros(4, dtype=torch.int32, device=cuda), 2)      # nobody signals
    with pytest.raises(RuntimeError):
        layer.check_status()
    own.reset_status()
    layer.check_status()


def test_add_rmsnorm_operands_in_place_or_apart(cuda):
    mem = torch.randn(16, 64, device=cuda).to(torch.bfloat16)
    x, t, w = mem[:4], mem[4:8], torch.ones(64, device=cuda, dtype=torch.bfloat16)
    h, y = x + t, ops.rmsnorm(x + t, w, 1e-5)
    for out, norm in ((mem[8:12], x), (t, mem[8:12]), (mem[8:12], t)):
        keep = mem.clone()
        _op().add_rmsnorm(x, t, out, norm, w, 1e-5)
        assert torch.equal(out, h) and torch.equal(norm, y)
        mem.copy_(keep)
    for out, norm in ((mem[2:6], mem[8:12]), (mem[8:12], mem[5:9]), (mem[8:12], mem[8:12]), (mem[8:12], mem[10:14])):
        with pytest.raises(RuntimeError):
            _op().add_rmsnorm(x, t, out, norm, w, 1e-5)
    with pytest.raises(RuntimeError):
        _op().add_rmsnorm(x, t, mem[8:12], mem[12:16], mem[9], 1e-5)


def test_rope_and_swiglu_refuse(cuda):
    qkv = torch.zeros(4, 256, device=cuda, dtype=torch.bfloat16)
    _op().rope_(qkv, 4, 2, 128, 1e4)
    for bad, seq, heads, hd in ((qkv, 4, 3, 128), (qkv, 0, 2, 128), (qkv, 4, 2, 12), (qkv, 4, -1, 128), (qkv.float(), 4, 2, 128),
                                (qkv[:, :128], 4, 1, 128), (qkv.view(-1), 4, 2, 128), (qkv.cpu(), 4, 2, 128),
                                (qkv.view(-1)[4:1012].view(4, 252), 4, 1, 128)):
        with pytest.raises(RuntimeError):
            _op().rope_(bad, seq, heads, hd, 1e4)
    gu, y = torch.zeros(4, 256, device=cuda, dtype=torch.bfloat16), torch.zeros(4, 128, device=cuda, dtype=torch.bfloat16)
    _op().swiglu(gu, y)
    for a, b in ((gu, y[:, :64]), (gu, y[:2]), (gu, y.half()), (gu.float(), y.float()), (gu, y.cpu()), (gu.view(-1), y), (gu[:, ::2], y),
                 (gu[:, :24].contiguous(), y[:, :12].contiguous()), (gu, gu.view(-1)[:512].view(4, 128)), (gu, gu.view(-1)[512:].view(4, 128))):
        with pytest.raises(RuntimeError):
            _op().swiglu(a, b)


def test_epilogue_gemms_refuse(cuda, impl):
    a, b, r, c = (torch.zeros(256, 256, device=cuda, dtype=torch.bfloat16) for _ in range(4))
    impl.gemm_add(a, b, r, c, 0)
    for bad in ((a[:, :128], b, r, c), (a, b.half(), r, c), (a, b, r[:128], c), (a, b, r, c[:128]), (a, b, r.half(), c), (a, b, r, c.float()),
                (a.cpu(), b, r, c), (a, b, r.cpu(), c), (a, b, r.t()[:, ::2], c), (a[:64], b, r, c)):
        with pytest.raises(RuntimeError):
            impl.gemm_add(*bad, 0)
    for algo in (-1, 1000):
        with pytest.raises(RuntimeError):
            impl.gemm_add(a, b, r, c, algo)
    y = torch.zeros(256, 128, device=cuda, dtype=torch.bfloat16)
    impl.gemm_swiglu(a, b, y)
    for bad in ((a[:64], b, y), (a, b[:128], y), (a, b, y[:64]), (a, b.half(), y), (a, b, y.half()), (a, b, y.cpu()), (a[:, :128], b, y),
                (a[:, :4].contiguous(), b[:, :4].contiguous(), y)):
        with pytest.raises(RuntimeError):
            impl.gemm_swiglu(*bad)
    impl.check_status()


def test_one_rank_layer_under_function_transforms(cuda):
    """vmap and forward mode over weights, which the fused kernels know nothing of, reach torch's operators."""
    from torch.autograd import forward_ad
    layer, x = _one_rank_layer(cuda)
    call = lambda **weights: torch.func.functional_call(layer, weights, (x,))
    wd = torch.stack([layer.wd.detach(), 2 * layer.wd.detach()])
    wgu = torch.stack([layer.wgu.detach(), layer.wgu.detach().flip(0)])
    with torch.no_grad():
        for name, many in (("wd", wd), ("wgu", wgu)):
            got = torch.vmap(lambda w: call(**{name: w}))(many)
            for i in range(2):
                ref = call(**{name: many[i]})
                assert (got[i] - ref).abs().max() <= 2.0 ** -6 * ref.abs().max()     # they round at different places
        tangent = torch.randn_like(layer.wd)
        with forward_ad.dual_level():
            out = forward_ad.unpack_dual(call(wd=forward_ad.make_dual(layer.wd.detach(), tangent)))
        # the output is linear in wd: its tangent is what the layer adds for the tangent's weights
        step = call(wd=tangent).float() - call(wd=torch.zeros_like(tangent)).float()
        assert out.tangent is not None and (out.tangent.float() - step).abs().max() <= 2.0 ** -6 * step.abs().max()


@pytest.mark.parametrize("T,hidden,ffn,adds,swiglus", [
    (2048, 2048, 512, (False, True), False), (2048, 2048, 1024, (False, True), True), (1920, 2048, 4096, (False, False), False),
    (2048, 4096, 2048, (True, True), True), (2048, 2048, 5120, (False, False), True), (2048, 8192, 5120, (True, True), True)])
def test_one_rank_layer_epilogues_by_size(cuda, T, hidden, ffn, adds, swiglus):
    """What the layer leaves to its GEMMs' epilogues, and that it computes the same either way."""
    from flashoverlap_b200.models import DecoderConfig, TPDecoderLayer
    cfg = DecoderConfig(hidden=hidden, ffn=ffn, n_heads=4, n_kv_heads=2)
    layer = TPDecoderLayer(cfg, 0, 1, 1, T, impl="fused", device=cuda)
    x = torch.randn(T, hidden, device=cuda).to(torch.bfloat16)
    with torch.no_grad():
        attn, act = x[:, :512].contiguous(), torch.randn(T, ffn, device=cuda).to(torch.bfloat16)
        assert (layer._adds(x, attn, layer.wo, norm=True), layer._adds(x, act, layer.wd)) == adds
        assert layer._swiglus(x) == swiglus
        y = layer(x)
        layer._fused_gemm = lambda *_: False
        plain = layer(x)
    assert (y - plain).abs().max() <= 2.0 ** -6 * plain.abs().max()       # they round at different places
    layer.check_status()
