"""Stand-alone operator entry points of the C ABI against the oracle's restatements."""
import numpy as np
import pytest

from lc0_b200 import _lib
from oracle import oracle

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

DT = {0: torch.float32, 1: torch.float16, 2: torch.bfloat16}


@pytest.mark.parametrize("prec", [0, 1, 2])
@pytest.mark.parametrize("n", [1, 3, 64, 257])
def test_expand_planes_bit_exact(lib, prec, n):
    rng = np.random.default_rng(n)
    masks = rng.integers(0, 2 ** 63, size=(n, 112), dtype=np.uint64) * np.uint64(2) + rng.integers(0, 2, size=(n, 112)).astype(np.uint64)
    values = rng.choice(np.array([1.0, 0.5, 0.25, 3.0, 99.0], np.float32), size=(n, 112))
    want = oracle.expand_planes(masks, values)
    dm = torch.from_numpy(masks.view(np.int64)).cuda()
    dv = torch.from_numpy(values).cuda()
    out = torch.zeros(n, 112, 64, dtype=DT[prec], device="cuda")
    _lib.check(lib.b200_op_expand_planes(dm.data_ptr(), dv.data_ptr(), n, out.data_ptr(), prec, None))
    torch.cuda.synchronize()
    assert np.array_equal(out.float().cpu().numpy(), want)  # all test values are exact in every type


def test_expand_planes_empty(lib):
    _lib.check(lib.b200_op_expand_planes(None, None, 0, None, 0, None))


@pytest.mark.parametrize("prec", [1, 2])
@pytest.mark.parametrize("shape", [(128, 64, 64), (64, 256, 512), (1000, 1024, 1024), (333, 200, 72),
                                   (8192, 3072, 1024), (4096, 1024, 1536), (130, 4096, 256), (2048, 32, 1024),
                                   # CTA-pair kernel with row / column tails (narrow last MMA tile) and few k-blocks
                                   # (four epilogue groups)
                                   (5000, 1312, 256), (3000, 2000, 1024), (2560, 1096, 320),
                                   # a last wave of at most half the CTA pairs: computed as half-width tiles
                                   (16384, 1024, 1024), (19200, 512, 256), (9600, 1024, 576)])
@pytest.mark.parametrize("act", [oracle.ACT_NONE, oracle.ACT_RELU_2, oracle.ACT_MISH])
def test_tensor_core_gemm(lib, prec, shape, act):
    M, N, K = shape
    torch.manual_seed(M + N + K)
    A = (torch.randn(M, K, device="cuda") * 0.5).to(DT[prec])
    W = (torch.randn(N, K, device="cuda") * (K ** -0.5)).to(DT[prec])
    b = torch.randn(N, device="cuda") * 0.1
    C = torch.zeros(M, N, dtype=DT[prec], device="cuda")
    _lib.check(lib.b200_op_gemm(A.data_ptr(), W.data_ptr(), b.data_ptr(), C.data_ptr(), M, N, K, act, prec, 1, None))
    torch.cuda.synchronize()
    ref = oracle.fc(A.float().cpu().numpy(), W.float().cpu().numpy().reshape(-1), b.cpu().numpy(), act, N)
    got = C.float().cpu().numpy()
    eps = 2.0 ** -10 if prec == 1 else 2.0 ** -7  # output rounding of the storage type
    assert np.all(np.abs(got - ref) <= eps * np.abs(ref) + 2e-3)


@pytest.mark.parametrize("prec", [0, 1, 2])
def test_fma_gemm(lib, prec):
    M, N, K = 77, 130, 45
    torch.manual_seed(0)
    A = (torch.randn(M, K, device="cuda")).to(DT[prec])
    W = (torch.randn(N, K, device="cuda") * 0.2).to(DT[prec])
    b = torch.randn(N, device="cuda")
    C = torch.zeros(M, N, dtype=DT[prec], device="cuda")
    _lib.check(lib.b200_op_gemm(A.data_ptr(), W.data_ptr(), b.data_ptr(), C.data_ptr(), M, N, K, oracle.ACT_SWISH, prec, 0, None))
    torch.cuda.synchronize()
    ref = oracle.fc(A.float().cpu().numpy(), W.float().cpu().numpy().reshape(-1), b.cpu().numpy(), oracle.ACT_SWISH, N)
    tol = {0: 1e-5, 1: 2e-3, 2: 1.6e-2}[prec]
    assert np.abs(C.float().cpu().numpy() - ref).max() <= tol * max(1.0, np.abs(ref).max())


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("M,N,K", [(1, 1, 1), (8, 64, 2048), (9, 65, 2047), (32, 4096, 256), (33, 63, 516), (64, 1024, 1024),
                                   (65, 130, 31), (200, 300, 1000), (1024, 1536, 128)])
def test_fma_gemm_tiles(lib, prec, M, N, K):
    """Edges of the FMA kernel's tiles (8 / 32 / 64 rows, 64 columns), K remainders, rows that cannot be read as 16-byte
    pieces, K ranges cut over a cluster."""
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    A = torch.randn(M, K, device="cuda", generator=g).to(DT[prec])
    W = torch.randn(N, K, device="cuda", generator=g).to(DT[prec])
    b = torch.randn(N, device="cuda", generator=g)
    C = torch.zeros(M, N, dtype=DT[prec], device="cuda")
    _lib.check(lib.b200_op_gemm(A.data_ptr(), W.data_ptr(), b.data_ptr(), C.data_ptr(), M, N, K, oracle.ACT_NONE, prec, 0, None))
    torch.cuda.synchronize()
    ref = A.double() @ W.double().T + b.double()
    mag = A.double().abs() @ W.double().abs().T + b.double().abs()
    # K + 1 roundings of sums no larger than mag, and the rounding of the storage type
    bound = (K + 2) * 2.0 ** -24 * mag + (2.0 ** -11 * ref.abs() + 2.0 ** -24 if prec == 1 else 0.0)
    assert torch.all((C.double() - ref).abs() <= bound), (C.double() - ref).abs().max().item()


@pytest.mark.parametrize("prec", [0, 1, 2])
@pytest.mark.parametrize("N,K", [(64, 100), (128, 255), (128, 256), (130, 511), (130, 512), (1024, 1024), (32, 1024), (256, 2047),
                                 (256, 2048), (64, 1022)])
def test_fma_gemm_rows_do_not_depend_on_their_number(lib, prec, N, K):
    """One summation order per (N, K): K in one, two, four or eight pieces, each by a CTA of its own (few tiles) or one after the
    other (many), tiles of 8, 32 and 64 rows."""
    g = torch.Generator(device="cuda").manual_seed(N + K)
    rows = 64 * 210 + 5
    A = torch.randn(rows, K, device="cuda", generator=g).to(DT[prec])
    W = torch.randn(N, K, device="cuda", generator=g).to(DT[prec])
    outs = []
    for M in (rows, 1, 5, 8, 9, 32, 33, 64, 65, 200, 3000):
        C = torch.zeros(M, N, dtype=DT[prec], device="cuda")
        _lib.check(lib.b200_op_gemm(A.data_ptr(), W.data_ptr(), None, C.data_ptr(), M, N, K, oracle.ACT_NONE, prec, 0, None))
        torch.cuda.synchronize()
        outs.append(C)
    for C in outs[1:]:
        assert torch.equal(C, outs[0][:C.shape[0]]), C.shape


def test_gemm_tc_rejects_fp32(lib):
    assert lib.b200_op_gemm(None, None, None, None, 128, 128, 64, 3, 0, 1, None) == _lib.ERR_UNSUPPORTED


def _f32_op(lib, A, W, bias, skip, conv, act=oracle.ACT_NONE, alpha=1.0):
    M, K, N = A.shape[0], A.shape[1], W.shape[-2]
    C = torch.full((M, N), 7.0, device="cuda")
    p = lambda t: None if t is None else t.data_ptr()
    _lib.check(lib.b200_op_gemm_f32(A.data_ptr(), A.stride(0), W.data_ptr(), p(bias), p(skip), C.data_ptr(), M, N, K, conv, act, alpha, None))
    return C


def _f32_want(A, W, conv):
    """Sums in 64 bits and the sums of the terms' magnitudes."""
    if not conv:
        return A.double() @ W.double().T, A.double().abs() @ W.double().abs().T
    x = A.double().view(-1, 8, 8, A.shape[1]).permute(0, 3, 1, 2)
    w = W.double().view(3, 3, W.shape[1], W.shape[2]).permute(2, 3, 0, 1)
    f = lambda a, b: torch.nn.functional.conv2d(a, b, padding=1).permute(0, 2, 3, 1).reshape(A.shape[0], -1)
    return f(x, w), f(x.abs(), w.abs())


@pytest.mark.parametrize("conv", [0, 1])
@pytest.mark.parametrize("shape", [(64, 8, 8), (64, 30, 72), (128, 64, 64), (192, 100, 112), (320, 130, 1024), (2048, 3072, 128),
                                   (64 * 210, 96, 200)])
def test_fp32_tensor_core_products(lib, conv, shape):
    """Three bf16 pieces per operand: edges of tiles (32 and 64 columns), of k-blocks and of board rows."""
    M, N, K = shape
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    A = torch.randn(M, K, device="cuda", generator=g)
    W = torch.randn(*((9, N, K) if conv else (N, K)), device="cuda", generator=g) * K ** -0.5
    b, skip = torch.randn(N, device="cuda", generator=g), torch.randn(M, N, device="cuda", generator=g)
    want, size = _f32_want(A, W, conv)
    got = _f32_op(lib, A, W, None, None, conv)
    # two truncating additions per 32 k, two rounded additions per 64 k, the pieces left out
    blocks = (9 if conv else 1) * ((K + 63) // 64)
    assert ((got.double() - want).abs() <= (4 + 2 * blocks + 1) * 2.0 ** -24 * size).all()
    got = _f32_op(lib, A, W, b, skip, conv, oracle.ACT_RELU, 0.5)
    want = 0.5 * torch.relu(want + b.double()) + skip.double()
    assert ((got.double() - want).abs() <= (4 + 2 * blocks + 4) * 2.0 ** -24 * (size + b.abs() + skip.abs())).all()
    whole = _f32_op(lib, A, W, b, None, conv)
    for rows in {64, M // 128 * 64 or 64}:  # a row's sum is the same among any number of rows
        assert torch.equal(_f32_op(lib, A[:rows], W, b, None, conv), whole[:rows])


@pytest.mark.parametrize("conv,N,K", [(0, 512, 1088), (0, 512, 1152), (0, 520, 1152), (0, 33, 2240), (0, 96, 2304), (0, 64, 4544), (0, 250, 4608),
                                      (1, 128, 64), (1, 96, 112), (1, 128, 128), (1, 256, 256), (1, 40, 448), (1, 512, 512), (1, 520, 512)])
def test_fp32_tensor_core_products_in_pieces_of_k(lib, conv, N, K):
    """Both sides of the lines where K is summed in two, four and eight pieces (18, 36 and 72 k-blocks, 512 columns): a CTA of a cluster
    for each piece on few rows, in turn on tiles of 32 and of 64 columns beyond; the same bits everywhere."""
    g = torch.Generator(device="cuda").manual_seed(N + K)
    A = torch.randn(64 * 150, K, device="cuda", generator=g)
    W = torch.randn(*((9, N, K) if conv else (N, K)), device="cuda", generator=g) * K ** -0.5
    b, skip = torch.randn(N, device="cuda", generator=g), torch.randn(A.shape[0], N, device="cuda", generator=g)
    plain = _f32_op(lib, A, W, None, None, conv)
    want, size = _f32_want(A[:640], W, conv)
    # as in test_fp32_tensor_core_products: a piece's two additions more are at most what its shorter chains save
    blocks = (9 if conv else 1) * ((K + 63) // 64)
    assert ((plain[:640].double() - want).abs() <= (4 + 2 * blocks + 1) * 2.0 ** -24 * size).all()
    whole = _f32_op(lib, A, W, b, skip, conv, oracle.ACT_RELU, 0.5)
    ref = torch.add(skip, torch.relu(plain + b), alpha=0.5)
    assert ((whole - ref).abs() <= 2.0 ** -22 * (ref.abs() + skip.abs())).all()  # the epilogue alone, contracted or not
    for rows in (64, 128, 192, 256, 640, 1600, 4096):
        assert torch.equal(_f32_op(lib, A[:rows], W, None, None, conv), plain[:rows])
        assert torch.equal(_f32_op(lib, A[:rows], W, b, skip[:rows], conv, oracle.ACT_RELU, 0.5), whole[:rows])
    A[3, 5], A[70, 1] = float("inf"), float("nan")  # computed again by FMAs, also from the sums of a cluster
    few, many = _f32_op(lib, A[:128], W, b, None, conv), _f32_op(lib, A, W, b, None, conv)[:128]
    assert torch.equal(few.nan_to_num(7e4, 8e4, 9e4), many.nan_to_num(7e4, 8e4, 9e4)) and not torch.isfinite(few[3]).any()


def _taps(A):
    """The rows of A that a 3x3 convolution reads, side by side: [M][9 * K]."""
    x = torch.nn.functional.pad(A.view(-1, 8, 8, A.shape[1]), (0, 0, 1, 1, 1, 1))
    return torch.cat([x[:, i:i + 8, j:j + 8] for i in range(3) for j in range(3)], 3).reshape(A.shape[0], -1).contiguous()


@pytest.mark.parametrize("conv,M,N,K", [(0, 256, 256, 64), (0, 1024, 1024, 256), (0, 512, 3072, 1024), (0, 512, 1024, 1536),
                                        (0, 128, 512, 4096), (1, 512, 128, 112), (1, 512, 128, 128), (1, 512, 256, 256)])
def test_fp32_tensor_core_products_against_the_fma_kernel(lib, conv, M, N, K):
    """Operands as the networks have them (weights of both signs; A of both or, behind a ReLU, of one): no further from sums in 64
    bits than the FMA kernel.  Operands that favour it (one sign, many decades, pieces that leave out the most): inside the
    bound of the header."""
    g = torch.Generator(device="cuda").manual_seed(N + K)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)
    wide = lambda *s: rnd(*s) * torch.exp(4 * rnd(*s))
    most = lambda *s: torch.full(s, 1 + 2.0 ** -8 - 2.0 ** -17 + 2.0 ** -23, device="cuda")
    blocks = (9 if conv else 1) * ((K + 63) // 64)
    shape = (9, N, K) if conv else (N, K)
    for of_a, of_w, network_like in ((rnd, rnd, True), (lambda *s: rnd(*s).relu(), rnd, True), (lambda *s: rnd(*s).abs(), lambda *s: rnd(*s).abs(), False),
                                     (wide, wide, False), (most, most, False)):
        A, W = of_a(M, K), of_w(*shape)
        a2, w2 = (_taps(A), W.permute(1, 0, 2).reshape(N, -1).contiguous()) if conv else (A, W)
        want, size = a2.double() @ w2.double().T, a2.double().abs() @ w2.double().abs().T
        got, fma = _f32_op(lib, A, W, None, None, conv).double(), torch.empty(M, N, device="cuda")
        assert ((got - want).abs() <= (7 + 1.34 * blocks) * 2.0 ** -24 * size).all()
        if network_like:
            _lib.check(lib.b200_op_gemm(a2.data_ptr(), w2.data_ptr(), None, fma.data_ptr(), M, N, a2.shape[1], oracle.ACT_NONE, 0, 0, None))
            torch.cuda.synchronize()
            assert (got - want).norm() <= (fma.double() - want).norm()


@pytest.mark.parametrize("conv", [0, 1])
def test_fp32_tensor_core_products_of_extreme_values(lib, conv):
    """Infinities, NaN, values that round to an infinite bf16 and values near the smallest normal: as the FMA kernel has them."""
    g = torch.Generator(device="cuda").manual_seed(5)
    A, W = torch.randn(128, 64, device="cuda", generator=g), torch.randn(*((9, 40, 64) if conv else (40, 64)), device="cuda", generator=g)
    A[3, 5], A[17, 6], A[40, 7], A[70, 8] = float("inf"), float("nan"), 3.4e38, -float("inf")
    A[100] *= 1e-35
    W[..., 8, :] = torch.tensor([1.0, 0.5] * 32, device="cuda")  # pieces 2 and 3 are zero
    W *= 0.25
    want, size = _f32_want(A, W, conv)
    want32 = want.float()
    got = _f32_op(lib, A, W, None, None, conv)
    assert torch.equal(got.isnan(), want32.isnan()) and torch.equal(got.isposinf(), want32.isposinf())
    assert torch.equal(got.isneginf(), want32.isneginf())
    ok = want32.isfinite()
    assert ((got.double() - want).abs()[ok] <= (20 * 2.0 ** -24 * size + 1e-37)[ok]).all()


def test_fp32_tensor_core_product_refuses(lib):
    a = torch.zeros(64 * 72, device="cuda").data_ptr()
    op = lambda A, lda, M, N, K, conv: lib.b200_op_gemm_f32(A, lda, a, None, None, a, M, N, K, conv, oracle.ACT_NONE, 1.0, None)
    assert op(a, 12, 8, 8, 12, 0) == _lib.ERR_UNSUPPORTED and op(a, 18, 8, 8, 16, 0) == _lib.ERR_UNSUPPORTED
    assert op(a + 4, 16, 8, 8, 16, 0) == _lib.ERR_UNSUPPORTED and op(a, 24, 64, 8, 16, 1) == _lib.ERR_UNSUPPORTED
    assert op(a, 16, 32, 8, 16, 1) == _lib.ERR_INVALID and op(None, 16, 8, 8, 16, 0) == _lib.ERR_INVALID


@pytest.mark.parametrize("prec", [0, 1, 2])
@pytest.mark.parametrize("C", [64, 256, 1024, 8192])
def test_layer_norm(lib, prec, C):
    rows = 130
    torch.manual_seed(C)
    x = torch.randn(rows, C, device="cuda").to(DT[prec])
    skip = torch.randn(rows, C, device="cuda").to(DT[prec])
    gam = torch.randn(C, device="cuda") * 0.1 + 1
    bet = torch.randn(C, device="cuda") * 0.1
    out = torch.zeros(rows, C, dtype=DT[prec], device="cuda")
    _lib.check(lib.b200_op_layer_norm(out.data_ptr(), x.data_ptr(), skip.data_ptr(), gam.data_ptr(), bet.data_ptr(),
                                      rows, C, 0.43, 1e-3, prec, None))
    torch.cuda.synchronize()
    ref = oracle.layer_norm(x.float().cpu().numpy(), 0.43, skip.float().cpu().numpy(), gam.cpu().numpy(),
                            bet.cpu().numpy(), 1e-3)
    tol = {0: 2e-5, 1: 4e-3, 2: 3e-2}[prec]
    assert np.abs(out.float().cpu().numpy() - ref).max() <= tol


def _policy_reference(q, k, w4):
    """Attention-policy tail restated with the oracle's table (network_blas.cc:850-914)."""
    from oracle import tables
    n, _, dm = q.shape
    logits = np.matmul(q, k.transpose(0, 2, 1)) / np.sqrt(np.float32(dm))
    off = np.einsum("njk,ik->nij", k[:, 56:64, :], w4)
    off[:, :3, :] += off[:, 3:4, :]
    promo = logits[:, 48:56, 56:64][:, :, :, None] + off[:, :3, :].transpose(0, 2, 1)[:, None, :, :]
    raw = np.concatenate([logits.reshape(n, 4096), promo.reshape(n, 192)], axis=1)
    pmap = tables.attn_policy_map()
    out = np.zeros((n, 1858), np.float32)
    out[:, pmap[pmap >= 0]] = raw[:, pmap >= 0]
    return out


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("n,dm", [(1, 64), (5, 96), (33, 256)])
def test_policy_attention_op(lib, prec, n, dm):
    torch.manual_seed(n * dm)
    q = torch.randn(n, 64, dm, device="cuda").to(DT[prec])
    k = torch.randn(n, 64, dm, device="cuda").to(DT[prec])
    w4 = torch.randn(4, dm, device="cuda") * 0.1
    scratch = torch.empty(n, 4096, device="cuda")
    pol = torch.zeros(n, 1858, device="cuda")
    _lib.check(lib.b200_op_policy_attention(q.data_ptr(), k.data_ptr(), w4.data_ptr(), dm, n, scratch.data_ptr(),
                                            pol.data_ptr(), prec, None))
    torch.cuda.synchronize()
    want = _policy_reference(q.float().cpu().numpy(), k.float().cpu().numpy(), w4.cpu().numpy())
    assert np.abs(pol.cpu().numpy() - want).max() <= 2e-4 * max(1.0, np.abs(want).max())


def _attention_reference(qkv, bias, n, heads, depth):
    """softmax(Q K^T / sqrt(depth) + bias) V per (position, head) in fp32 (network_blas.cc:352-439)."""
    e = heads * depth
    x = qkv.float().reshape(n, 64, 3, heads, depth)
    q, k, v = (x[:, :, i].permute(0, 2, 1, 3) for i in range(3))  # [n][heads][64][depth]
    s = torch.matmul(q, k.transpose(-1, -2)) / depth ** 0.5
    if bias is not None:
        s = s + bias.float().reshape(n, heads, 64, 64)
    p = torch.softmax(s, dim=-1)
    return torch.matmul(p, v).permute(0, 2, 1, 3).reshape(n * 64, e)


@pytest.mark.parametrize("variant", [0, 1])
@pytest.mark.parametrize("prec", [1, 2])
@pytest.mark.parametrize("n,heads,depth,with_bias", [(1, 4, 32, True), (7, 32, 32, True), (3, 8, 64, False),
                                                     (150, 8, 32, True), (40, 6, 64, True), (2, 1, 32, False)])
def test_attention_op(lib, variant, prec, n, heads, depth, with_bias):
    """Both attention kernels against an fp32 reference on the fused Q|K|V layout the network uses; the
    persistent TMA kernel (variant 1) walks several items per CTA at the larger sizes."""
    torch.manual_seed(n * heads + depth)
    e = heads * depth
    qkv = torch.randn(n * 64, 3 * e, device="cuda").to(DT[prec])
    bias = (torch.randn(n, heads, 64, 64, device="cuda") * 2).to(DT[prec]) if with_bias else None
    out = torch.zeros(n * 64, e, device="cuda", dtype=DT[prec])
    esz = 2
    _lib.check(lib.b200_op_attention(qkv.data_ptr(), qkv.data_ptr() + e * esz, qkv.data_ptr() + 2 * e * esz, 3 * e,
                                     bias.data_ptr() if with_bias else None, out.data_ptr(), e, n, heads, depth, prec,
                                     variant, None))
    torch.cuda.synchronize()
    want = _attention_reference(qkv, bias, n, heads, depth)
    tol = 4e-3 if prec == 1 else 3e-2  # probabilities and outputs are rounded to 16 bits (11 / 8 significant bits)
    assert (out.float() - want).abs().max().item() <= tol * max(1.0, want.abs().max().item())


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("heads,depth,pad,shift", [(3, 32, 0, 0), (3, 32, 4, 4), (3, 32, 1, 0), (3, 32, 4, 1), (2, 30, 0, 0),
                                                   (2, 4, 0, 0), (1, 2, 0, 0), (1, 128, 0, 0)])
def test_attention_op_rows_in_pieces_of_four(lib, prec, heads, depth, pad, shift):
    """Rows that start on four-number boundaries and rows that do not (odd leading dimension, shifted base, odd head width).
    fp32 bound: each score carries (depth + 3) roundings of at most the sum of |q||k|, doubled by the normalisation, the weighted
    sum 64 more and the exponential a few."""
    torch.manual_seed(depth + pad)
    n, e = 2, heads * depth
    dt = torch.float32 if prec == 0 else DT[prec]
    ld = 3 * e + pad
    store = torch.randn(n * 64 * ld + shift, device="cuda").to(dt)
    qkv = store[shift:].reshape(n * 64, ld)[:, :3 * e]
    bias = torch.randn(n, heads, 64, 64, device="cuda").to(dt)
    out = torch.zeros(n * 64, e, device="cuda", dtype=dt)
    esz = out.element_size()
    base = store.data_ptr() + shift * esz
    _lib.check(lib.b200_op_attention(base, base + e * esz, base + 2 * e * esz, ld, bias.data_ptr(), out.data_ptr(), e, n, heads,
                                     depth, prec, 0, None))
    torch.cuda.synchronize()
    q, k, v = (t.permute(0, 2, 1, 3) for t in qkv.double().reshape(n, 64, 3, heads, depth).unbind(2))
    s = torch.matmul(q, k.transpose(-1, -2)) / depth ** 0.5 + bias.double()
    want = torch.matmul(torch.softmax(s, -1), v).permute(0, 2, 1, 3).reshape(n * 64, e)
    size = (torch.matmul(q.abs(), k.abs().transpose(-1, -2)) / depth ** 0.5 + bias.double().abs()).max().item()
    tol = (2 * (depth + 3) * size + 64 + 16) * 2.0 ** -24 * v.abs().max().item() if prec == 0 else 4e-3 * max(1.0, want.abs().max().item())
    assert (out.double() - want).abs().max().item() <= tol


def test_attention_op_variants_agree(lib):
    """The FMA kernel and the persistent TMA kernel on the same 16-bit inputs."""
    torch.manual_seed(5)
    n, heads, depth = 64, 32, 32
    e = heads * depth
    qkv = torch.randn(n * 64, 3 * e, device="cuda").half()
    bias = torch.randn(n, heads, 64, 64, device="cuda").half()
    outs = []
    for variant in (0, 1):
        out = torch.zeros(n * 64, e, device="cuda", dtype=torch.float16)
        _lib.check(lib.b200_op_attention(qkv.data_ptr(), qkv.data_ptr() + e * 2, qkv.data_ptr() + 4 * e, 3 * e,
                                         bias.data_ptr(), out.data_ptr(), e, n, heads, depth, 1, variant, None))
        outs.append(out.float())
    torch.cuda.synchronize()
    assert (outs[0] - outs[1]).abs().max().item() <= 4e-3


def test_attention_op_rejects_fp32_tensor_core_variants(lib):
    assert lib.b200_op_attention(None, None, None, 96, None, None, 32, 0, 1, 32, 0, 1, None) == _lib.ERR_UNSUPPORTED


# ---- folded-LayerNorm epilogues of the tensor-core product (b200_op_gemm_ex) -------------------------------------
def _desc(**kw):
    d = _lib.GemmDesc()
    d.scale, d.alpha = 1.0, 1.0
    for k, v in kw.items():
        setattr(d, k, v.data_ptr() if hasattr(v, "data_ptr") else v)
    return d


def _planted_rows(M):
    """Row classes of the epilogue tests: rows whose mean is many standard deviations away from zero, rows with one
    channel at 3e3 or 1e4, and ordinary rows."""
    r = np.arange(M)
    return {"shifted": r[r % 7 == 3], "outlier3e3": r[r % 11 == 5], "outlier1e4": r[r % 13 == 8]}


def _fold(W, b, gamma, beta, dt):
    """What the loader does for a product that consumes a folded LayerNorm: W * gamma rounded to the storage type,
    its row sums, and beta . W^T + b."""
    Wg = (W * gamma[None, :]).to(dt)
    colsum = Wg.float().sum(dim=1).contiguous()
    bias = (b.double() + (W.double() * beta.double()[None, :]).sum(dim=1)).float().contiguous()
    return Wg.contiguous(), colsum, bias


@pytest.mark.parametrize("prec,M,shift", [(1, 65536, 100.0), (2, 8192 + 77, 10.0)])
def test_folded_layer_norm_epilogues_against_oracle(lib, prec, M, shift):
    """The three epilogue forms an encoder layer uses, chained as in the layer, at the row count of batch 1024:
      1. u  = alpha * (A0 W0^T + b0) + R            with per-row (sum, sum of squares) of u accumulated by atomics
      2. h  = relu2(LN(u) W1^T + b1)                LayerNorm folded: row scale and rank-1 correction from the statistics
      3. u2 = alpha * (h W2^T + b2) + LN(u)         the residual normalised on the fly, statistics of u2 again
    against oracle.fc / oracle.layer_norm (fully_connected_layer.cc:50-106, backends/blas/encoder.h:29-78) on a
    sample of rows that contains every planted row class.  The row statistics are sums of the unrounded outputs while
    the consumer reads the rounded ones, so bf16 (spacing 0.5 at 100) gets a smaller row shift than fp16."""
    dt = DT[prec]
    E, F = 1024, 1536
    alpha, eps_ln = 0.43, 1e-3
    g = torch.Generator(device="cuda").manual_seed(M + prec)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)
    A0 = (rnd(M, E) * 0.5).to(dt)
    W0 = (rnd(E, E) * E ** -0.5).to(dt)
    b0 = rnd(E) * 0.1
    R = rnd(M, E)
    rows = _planted_rows(M)
    R[torch.from_numpy(rows["shifted"]).cuda()] += shift
    R[torch.from_numpy(rows["outlier3e3"]).cuda(), 5] = 3000.0
    R[torch.from_numpy(rows["outlier1e4"]).cuda(), 700] = -10000.0
    R = R.to(dt)
    gamma = 1 + rnd(E) * 0.1
    beta = rnd(E) * 0.1
    W1 = rnd(F, E) * E ** -0.5
    b1 = rnd(F) * 0.1
    W2 = (rnd(E, F) * F ** -0.5).to(dt)
    b2 = rnd(E) * 0.1
    W1g, cs1, b1f = _fold(W1, b1, gamma, beta, dt)

    u = torch.zeros(M, E, dtype=dt, device="cuda")
    st1 = torch.zeros(M, 2, device="cuda", dtype=torch.float64)
    _lib.check(lib.b200_op_gemm_ex(_desc(A=A0, W=W0, bias=b0, C=u, M=M, N=E, K=E, precision=prec, alpha=alpha,
                                         res=R, out_stats=st1), None))
    h = torch.zeros(M, F, dtype=dt, device="cuda")
    _lib.check(lib.b200_op_gemm_ex(_desc(A=u, W=W1g, bias=b1f, C=h, M=M, N=F, K=E, precision=prec,
                                         activation=oracle.ACT_RELU_2, a_stats=st1, colsum=cs1, a_inv_c=1.0 / E,
                                         a_eps=eps_ln), None))
    u2 = torch.zeros(M, E, dtype=dt, device="cuda")
    st2 = torch.zeros(M, 2, device="cuda", dtype=torch.float64)
    _lib.check(lib.b200_op_gemm_ex(_desc(A=h, W=W2, bias=b2, C=u2, M=M, N=E, K=F, precision=prec, alpha=alpha,
                                         res=u, res_stats=st1, res_gamma=gamma, res_beta=beta, res_inv_c=1.0 / E,
                                         res_eps=eps_ln, out_stats=st2), None))
    torch.cuda.synchronize()

    rng = np.random.default_rng(7)
    sample = np.unique(np.concatenate([rows["shifted"][:96], rows["outlier3e3"][:64], rows["outlier1e4"][:64],
                                       rng.integers(0, M, 256), [0, M - 1]]))
    sel = torch.from_numpy(sample).cuda()
    f = lambda t: (t if t.dtype == torch.float64 else t.float()).cpu().numpy()
    rt = 2.0 ** -10 if prec == 1 else 2.0 ** -7  # output rounding of the storage type
    # 1: product + plain residual + statistics
    u_ref = alpha * oracle.fc(f(A0[sel]), f(W0).reshape(-1), f(b0), oracle.ACT_NONE, E) + f(R[sel])
    assert np.all(np.abs(f(u[sel]) - u_ref) <= rt * np.abs(u_ref) + 2e-3)
    s_ref = np.stack([u_ref.sum(-1, dtype=np.float64), (u_ref.astype(np.float64) ** 2).sum(-1)], 1)
    mag = np.stack([np.abs(u_ref).sum(-1, dtype=np.float64), s_ref[:, 1]], 1)  # what the fp32 partial sums add up
    assert np.all(np.abs(f(st1[sel]) - s_ref) <= 2e-5 * mag + 1e-3)
    # 2: folded LayerNorm of the stored (rounded) u, two-pass in the oracle
    un = f(u[sel])
    x = oracle.layer_norm(un, 1.0, None, np.ones(E, np.float32), np.zeros(E, np.float32), eps_ln)
    h_ref = oracle.fc(x, f(W1g).reshape(-1), f(b1f), oracle.ACT_RELU_2, F)
    # Rows shifted by `shift` standard deviations: the folded form computes LN(u) W^T as rstd * (u W'^T - mean * colsum),
    # two terms of size |mean| * |colsum| that cancel; the tensor core accumulates the first one at that size, so the
    # pre-activation loses about 1e-4 * shift (fp16; more in bf16, whose statistics are also sums of the unrounded
    # values while the product reads the rounded ones), and relu^2 turns it into 2 * sqrt(h) times that.
    is_shifted = np.isin(sample, rows["shifted"])[:, None]
    per_shift = 2e-4 if prec == 1 else 1e-3

    def worst(got, ref, floor):
        extra = np.where(is_shifted, per_shift * shift * (1 + 2 * np.sqrt(np.abs(ref))), 0.0)
        err = np.abs(got - ref) - (rt * np.abs(ref) + floor + extra)
        r, c = np.unravel_index(err.argmax(), err.shape)
        cls = [k for k, v in rows.items() if sample[r] in v] or ["ordinary"]
        return err.max(), "excess %.3g at row %d (%s) column %d: got %.6g, reference %.6g" % (
            err.max(), sample[r], "+".join(cls), c, got[r, c], ref[r, c])

    e, msg = worst(f(h[sel]), h_ref, 3e-3)
    assert e <= 0, "folded LayerNorm product: " + msg
    # 3: residual normalised on the fly
    ln_u = oracle.layer_norm(un, 1.0, None, f(gamma), f(beta), eps_ln)
    u2_ref = alpha * oracle.fc(f(h[sel]), f(W2).reshape(-1), f(b2), oracle.ACT_NONE, E) + ln_u
    e, msg = worst(f(u2[sel]), u2_ref, 3e-3)
    assert e <= 0, "normalised residual: " + msg
    s2_ref = np.stack([u2_ref.sum(-1, dtype=np.float64), (u2_ref.astype(np.float64) ** 2).sum(-1)], 1)
    mag2 = np.stack([np.abs(u2_ref).sum(-1, dtype=np.float64), s2_ref[:, 1]], 1)
    # u2_ref is built from the rounded h and u, the kernel's sums from its own unrounded values: the storage
    # type's rounding, not the summation, bounds the difference
    assert np.all(np.abs(f(st2[sel]) - s2_ref) <= 4 * rt * mag2 + 1e-2)


@pytest.mark.parametrize("whole_tiles", [0, 1])
def test_second_output_of_the_pair_kernel_with_folded_input(lib, whole_tiles):
    """Q, K, V and the smolgen compression from one launch (columns from n_split on go to a second matrix through a
    narrow last tile), with the LayerNorm of the input folded in, at the row count of batch 1024."""
    M, E, N, hc = 65536, 1024, 3072, 32
    g = torch.Generator(device="cuda").manual_seed(11)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)
    u = (rnd(M, E) * 2 + 0.5).half()
    gamma, beta = 1 + rnd(E) * 0.1, rnd(E) * 0.1
    W = rnd(N + hc, E) * E ** -0.5
    b = torch.cat([rnd(N) * 0.1, torch.zeros(hc, device="cuda")])
    Wg, cs, bf = _fold(W, b, gamma, beta, torch.float16)
    uf = u.double()
    stats = torch.stack([uf.sum(1), (uf * uf).sum(1)], 1).contiguous()
    C = torch.zeros(M, N, dtype=torch.float16, device="cuda")
    C2 = torch.zeros(M, hc, dtype=torch.float16, device="cuda")
    _lib.check(lib.b200_op_gemm_ex(_desc(A=u, W=Wg, bias=bf, C=C, M=M, N=N + hc, K=E, precision=1, a_stats=stats,
                                         colsum=cs, a_inv_c=1.0 / E, a_eps=1e-3, C2=C2, ldc2=hc, n_split=N,
                                         whole_tiles=whole_tiles), None))
    torch.cuda.synchronize()
    sample = np.unique(np.concatenate([np.random.default_rng(3).integers(0, M, 300), [0, 127, 128, M - 129, M - 1]]))
    sel = torch.from_numpy(sample).cuda()
    f = lambda t: t.float().cpu().numpy()
    x = oracle.layer_norm(f(u[sel]), 1.0, None, np.ones(E, np.float32), np.zeros(E, np.float32), 1e-3)
    ref = oracle.fc(x, f(Wg).reshape(-1), f(bf), oracle.ACT_NONE, N + hc)
    got = np.concatenate([f(C[sel]), f(C2[sel])], 1)
    assert np.all(np.abs(got - ref) <= 2.0 ** -10 * np.abs(ref) + 3e-3)


@pytest.mark.parametrize("prec", [1, 2])
@pytest.mark.parametrize("form", ["res act", "stats act", "norm res", "norm res stats"])
@pytest.mark.parametrize("M,N,K", [(8192, 1024, 512), (8200, 1000, 520), (8192, 1024, 576), (8200, 1000, 584), (8200, 1000, 768),
                                   (8192, 1024, 776), (8200, 1000, 1024), (8192, 1024, 1032)])
def test_forms_of_the_pair_kernel_that_no_layer_has(lib, prec, form, M, N, K):
    """Residual or statistics beside an activation or a folded LayerNorm of A: both sides of the lines between two and four
    groups of epilogue warps and the forms of issue (8, 9, 12 and 16 k-blocks), ragged rows, columns and k-blocks."""
    dt = DT[prec]
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)
    A, W = (rnd(M, K) + 0.5).to(dt), (rnd(N, K) * K ** -0.5).to(dt)
    b, cs = rnd(N) * 0.1, W.float().sum(1).contiguous()
    a64 = A.double()
    C, out_st = torch.zeros(M, N, dtype=dt, device="cuda"), torch.zeros(M, 2, device="cuda", dtype=torch.float64)
    kw = dict(A=A, W=W, bias=b, C=C, M=M, N=N, K=K, precision=prec, activation=oracle.ACT_NONE)
    ref = a64 @ W.double().T
    if "norm" in form:
        st_a = torch.stack([a64.sum(1), (a64 * a64).sum(1)], 1).contiguous()
        kw.update(a_stats=st_a, colsum=cs, a_inv_c=1.0 / K, a_eps=1e-3)
        ref = (ref - a64.mean(1, keepdim=True) * cs.double()) * (a64.var(1, unbiased=False, keepdim=True) + 1e-3).rsqrt()
    ref = ref + b.double()
    if "act" in form:
        kw.update(activation=oracle.ACT_SWISH)
        ref = ref * torch.sigmoid(ref)
    if "res" in form:
        R = rnd(M, N).to(dt)
        kw.update(res=R, alpha=0.43)
        ref = 0.43 * ref + R.double()
    if "stats" in form:
        kw.update(out_stats=out_st)
    _lib.check(lib.b200_op_gemm_ex(_desc(**kw), None))
    torch.cuda.synchronize()
    # as in test_products_of_few_rows: rounding of the storage type, fp32 sums, the fast exponential
    rt = 2.0 ** -10 if prec == 1 else 2.0 ** -7
    assert torch.all((C.double() - ref).abs() <= rt * ref.abs() + 1e-3), (C.double() - ref).abs().max().item()
    if "stats" in form:
        s_ref = torch.stack([ref.sum(1), (ref * ref).sum(1)], 1)
        mag = torch.stack([ref.abs().sum(1), s_ref[:, 1]], 1)
        assert torch.all((out_st - s_ref).abs() <= 1e-3 * mag + 1e-3)


@pytest.mark.parametrize("prec", [1, 2])
@pytest.mark.parametrize("M,N,K", [(1, 8, 8), (1, 256, 2048), (3, 8192, 256), (7, 40, 72), (63, 1024, 1024), (64, 1536, 1024),
                                   (65, 1024, 1536), (130, 200, 624), (384, 1024, 1024), (1000, 1858, 64),
                                   (1537, 128, 512)])
def test_products_of_few_rows(lib, prec, M, N, K):
    """The split-K kernel at the edges of its tiles (64 / 128 rows, 32 / 64 / 128 columns, K remainders, columns that are no
    multiple of eight) with every epilogue form: folded LayerNorm of A, activation, residual normalised on the fly,
    row statistics.  fp32 reference of the same arithmetic on the stored operands."""
    dt = DT[prec]
    g = torch.Generator(device="cuda").manual_seed(M * 7 + N + K)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)
    A = (rnd(M, K) + 0.5).to(dt)
    W = (rnd(N, K) * K ** -0.5).to(dt)
    b, cs = rnd(N) * 0.1, W.float().sum(1).contiguous()
    a64 = A.double()
    st_a = torch.stack([a64.sum(1), (a64 * a64).sum(1)], 1).contiguous()
    C = torch.zeros(M, N, dtype=dt, device="cuda")
    out_st = torch.zeros(M, 2, device="cuda", dtype=torch.float64)
    kw = dict(A=A, W=W, bias=b, C=C, M=M, N=N, K=K, precision=prec, activation=oracle.ACT_SWISH, out_stats=out_st,
              a_stats=st_a, colsum=cs, a_inv_c=1.0 / K, a_eps=1e-3, alpha=0.43)
    mean = a64.mean(1, keepdim=True)
    rstd = (a64.var(1, unbiased=False, keepdim=True) + 1e-3).rsqrt()
    v = rstd * (a64 @ W.double().T - mean * cs.double()) + b.double()
    ref = 0.43 * v * torch.sigmoid(v)
    if N % 8 == 0:
        R = (rnd(M, N) * 2 + 1).to(dt)
        r64 = R.double()
        st_r = torch.stack([r64.sum(1), (r64 * r64).sum(1)], 1).contiguous()
        gamma, beta = 1 + rnd(N) * 0.1, rnd(N) * 0.1
        kw.update(res=R, res_stats=st_r, res_gamma=gamma, res_beta=beta, res_inv_c=1.0 / N, res_eps=1e-3)
        rn = (r64 - r64.mean(1, keepdim=True)) * (r64.var(1, unbiased=False, keepdim=True) + 1e-3).rsqrt()
        ref = ref + rn * gamma.double() + beta.double()
    else:
        kw.update(alpha=1.0)
        ref = ref / 0.43
    if N % 8:  # the folded forms need rows that TMA can describe elsewhere in the schedule; plain epilogue here
        for k in ("out_stats", "a_stats", "colsum"):
            kw.pop(k)
        v = a64 @ W.double().T + b.double()
        ref = v * torch.sigmoid(v)
    _lib.check(lib.b200_op_gemm_ex(_desc(**kw), None))
    torch.cuda.synchronize()
    # output rounding of the storage type; fp32 accumulation of K products of magnitude rstd * |A| * |W|, of which the
    # LayerNorm correction cancels the mean's part: a few 1e-5 at most, 2e-4 with the fast exponential of the activation
    rt = 2.0 ** -10 if prec == 1 else 2.0 ** -7
    got = C.double()
    assert torch.all((got - ref).abs() <= rt * ref.abs() + 1e-3), (got - ref).abs().max().item()
    if "out_stats" in kw:
        s_ref = torch.stack([ref.sum(1), (ref * ref).sum(1)], 1)
        mag = torch.stack([ref.abs().sum(1), s_ref[:, 1]], 1)
        assert torch.all((out_st - s_ref).abs() <= 1e-3 * mag + 1e-3)


@pytest.mark.parametrize("prec", [1, 2])
@pytest.mark.parametrize("N,K", [(256, 2048), (1024, 1024), (40, 72), (1858, 2048), (8192, 256)])
def test_tensor_core_gemm_rows_do_not_depend_on_their_number(lib, prec, N, K):
    """One result of a row for all numbers of rows below 64 and one from 64 on, whichever kernel and tile they go to."""
    g = torch.Generator(device="cuda").manual_seed(N + K)
    A = torch.randn(6000, K, device="cuda", generator=g).to(DT[prec])
    W = (torch.randn(N, K, device="cuda", generator=g) * K ** -0.5).to(DT[prec])
    b = torch.randn(N, device="cuda", generator=g)
    for sizes in ((63, 1, 2, 8, 33), (6000, 64, 65, 200, 700, 2048)):
        outs = []
        for M in sizes:
            C = torch.zeros(M, N, dtype=DT[prec], device="cuda")
            _lib.check(lib.b200_op_gemm(A.data_ptr(), W.data_ptr(), b.data_ptr(), C.data_ptr(), M, N, K, oracle.ACT_MISH, prec, 1, None))
            outs.append(C)
        for C in outs[1:]:
            assert torch.equal(C, outs[0][:C.shape[0]]), C.shape


@pytest.mark.parametrize("M", [1, 65, 1000, 40000])
def test_gemm_ex_refuses_rows_its_epilogue_cannot_address(lib, M):
    """Residuals, statistics and second outputs whose rows do not lie on 16-byte boundaries are refused on the host, whichever
    kernel the number of rows would have gone to (the split-K kernel's 16-byte loads would be misaligned)."""
    N, K = 20, 64
    half = lambda *s: torch.zeros(*s, dtype=torch.float16, device="cuda")
    A, W, C, R = half(M, K), half(512, K), half(M, 528), half(M * 528 + 8)
    st = torch.zeros(M, 2, dtype=torch.float64, device="cuda")
    cs = torch.zeros(512, device="cuda")
    base = dict(A=A, W=W, C=C, M=M, N=N, K=K, precision=1, activation=oracle.ACT_NONE, ldc=24)
    good = dict(base, res=R, ldres=24)
    _lib.check(lib.b200_op_gemm_ex(_desc(**good), None))
    _lib.check(lib.b200_op_gemm_ex(_desc(**dict(base, ldc=0)), None))  # plain products go through plain stores
    for bad in (dict(good, ldres=20), dict(good, ldres=0), dict(good, res=R.data_ptr() + 2), dict(good, ldc=20),
                dict(good, C=C.data_ptr() + 8), dict(base, ldc=20, out_stats=st),
                dict(base, ldc=20, a_stats=st, colsum=cs, a_inv_c=1.0 / K)):
        assert lib.b200_op_gemm_ex(_desc(**bad), None) == _lib.ERR_CUDA
    for bad in (dict(base, N=288, n_split=256, ldc=260, C2=R, ldc2=32), dict(base, N=288, n_split=256, ldc=256, C2=R, ldc2=36)):
        assert lib.b200_op_gemm_ex(_desc(**bad), None) == _lib.ERR_UNSUPPORTED
    torch.cuda.synchronize()


@pytest.mark.parametrize("prec", [1, 2])
@pytest.mark.parametrize("group,M,N", [(1, 1, 256), (1, 63, 8192), (1, 65, 40), (2, 2, 64), (2, 66, 200), (4, 4, 4096), (4, 68, 72),
                                       (8, 8, 128), (8, 200, 96), (16, 16, 4096), (16, 80, 65), (32, 32, 4096), (32, 96, 100),
                                       (32, 256, 4096)])
def test_layer_norm_inside_a_product(lib, prec, group, M, N):
    """Vectors of 1 to 32 rows (sums over lanes, over one warp, over several), the last tile full or not, columns that are no
    multiple of the tile or of eight; one vector far from zero mean, one almost constant."""
    dt = DT[prec]
    g = torch.Generator(device="cuda").manual_seed(group * 1000 + M + N)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)
    vec = M // group
    x = rnd(vec, group * 256)
    x[0] += 20.0
    x[-1] *= 1e-2
    x = x.to(dt)
    gamma, beta = 1 + 0.2 * rnd(group * 256), 0.2 * rnd(group * 256)
    W, b = (rnd(N, 256) / 16).to(dt), 0.1 * rnd(N)
    C = torch.zeros(M, N, dtype=dt, device="cuda")
    _lib.check(lib.b200_op_gemm_ln(x.data_ptr(), gamma.data_ptr(), beta.data_ptr(), group, 1e-3, W.data_ptr(), b.data_ptr(),
                                   C.data_ptr(), M, N, oracle.ACT_NONE, prec, None))
    x64 = x.double()
    xn = (x64 - x64.mean(1, keepdim=True)) * (x64.var(1, unbiased=False, keepdim=True) + 1e-3).rsqrt()
    xn = (xn * gamma.double() + beta.double()).reshape(M, 256)
    ref = xn @ W.double().T + b.double()
    mag = xn.abs() @ W.double().abs().T
    # the normalised rows are rounded to the storage type once and so is the result; in fp32, mean and variance of up to 8192
    # values whose mean is 20 deviations away lose 2^-24 * 20 * (a few) of a deviation
    u = 2.0 ** -11 if prec == 1 else 2.0 ** -8
    assert torch.all((C.double() - ref).abs() <= (u + 1e-5) * mag + u * ref.abs() + 1e-4), (C.double() - ref).abs().max().item()


def test_layer_norm_inside_a_product_refuses_other_shapes(lib):
    x = torch.zeros(64, 256, dtype=torch.float16, device="cuda")
    v = torch.zeros(64 * 256, device="cuda")
    op = lambda group, M, prec, off=0: lib.b200_op_gemm_ln(x.data_ptr() + off, v.data_ptr(), v.data_ptr(), group, 1e-3, x.data_ptr(),
                                                           None, x.data_ptr(), M, 64, oracle.ACT_NONE, prec, None)
    for args in ((1, 4, 0), (3, 6, 1), (64, 64, 1), (0, 4, 1), (8, 12, 1), (1, 4, 1, 8)):
        assert op(*args) == _lib.ERR_UNSUPPORTED


@pytest.mark.parametrize("prec", [1, 2])
@pytest.mark.parametrize("M,rest", [(1, 8), (63, 32), (64, 256), (65, 200), (130, 40), (400, 104)])
def test_second_output_of_products_of_few_rows(lib, prec, M, rest):
    """Columns beyond n_split go to the second matrix, with the LayerNorm of the input folded in; widths that end inside a tile and
    row counts that end inside a tile.  Neither matrix is written beyond its columns."""
    dt, N, K = DT[prec], 512, 320
    g = torch.Generator(device="cuda").manual_seed(M + rest)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)
    A, W, b = (rnd(M, K) + 0.5).to(dt), (rnd(N + rest, K) * K ** -0.5).to(dt), 0.1 * rnd(N + rest)
    a64 = A.double()
    st = torch.stack([a64.sum(1), (a64 * a64).sum(1)], 1).contiguous()
    cs = W.float().sum(1).contiguous()
    C, C2 = torch.full((M, N + 8), 7.0, dtype=dt, device="cuda"), torch.full((M, rest + 8), 7.0, dtype=dt, device="cuda")
    _lib.check(lib.b200_op_gemm_ex(_desc(A=A, W=W, bias=b, C=C, M=M, N=N + rest, K=K, ldc=N + 8, precision=prec, a_stats=st, colsum=cs,
                                         activation=oracle.ACT_NONE, a_inv_c=1.0 / K, a_eps=1e-3, C2=C2, ldc2=rest + 8,
                                         n_split=N), None))
    rstd = (a64.var(1, unbiased=False, keepdim=True) + 1e-3).rsqrt()
    ref = rstd * (a64 @ W.double().T - a64.mean(1, keepdim=True) * cs.double()) + b.double()
    got = torch.cat([C[:, :N], C2[:, :rest]], 1).double()
    u = 2.0 ** -11 if prec == 1 else 2.0 ** -8
    # fp32: K products and the mean's correction, each at most rstd * (|A| |W|), a few roundings of it
    mag = rstd * (a64.abs() @ W.double().abs().T)
    assert torch.all((got - ref).abs() <= u * ref.abs() + 1e-5 * mag + 1e-6), (got - ref).abs().max().item()
    assert torch.all(C[:, N:] == 7) and torch.all(C2[:, rest:] == 7)


@pytest.mark.parametrize("M,N,ldc", [(1, 8, 9), (65, 129, 131), (200, 1858, 1858), (64, 64, 65)])
def test_products_of_few_rows_into_unaligned_rows(lib, M, N, ldc):
    """Output rows that are no 16-byte pieces: element stores, nothing beyond the columns."""
    K = 136
    g = torch.Generator(device="cuda").manual_seed(M + N)
    A = torch.randn(M, K, device="cuda", generator=g).half()
    W = (torch.randn(N, K, device="cuda", generator=g) * K ** -0.5).half()
    C = torch.full((M, ldc), 7.0, dtype=torch.float16, device="cuda")
    _lib.check(lib.b200_op_gemm_ex(_desc(A=A, W=W, C=C, M=M, N=N, K=K, ldc=ldc, precision=1, activation=oracle.ACT_NONE), None))
    ref = A.double() @ W.double().T
    mag = A.double().abs() @ W.double().abs().T
    assert torch.all((C[:, :N].double() - ref).abs() <= 2.0 ** -11 * ref.abs() + (K + 2) * 2.0 ** -24 * mag + 2.0 ** -24)
    assert torch.all(C[:, N:] == 7)


def test_gemm_ex_rejects_inconsistent_descriptions(lib):
    a = torch.zeros(256, 64, dtype=torch.float16, device="cuda")
    st = torch.zeros(256, 2, device="cuda", dtype=torch.float64)
    assert lib.b200_op_gemm_ex(_desc(A=a, W=a, C=a, M=256, N=64, K=64, precision=0), None) == _lib.ERR_UNSUPPORTED
    assert lib.b200_op_gemm_ex(_desc(A=a, W=a, C=a, M=256, N=64, K=64, precision=1, a_stats=st), None) == \
        _lib.ERR_UNSUPPORTED  # statistics without column sums
    assert lib.b200_op_gemm_ex(_desc(A=a, W=a, C=a, M=256, N=64, K=64, precision=1, C2=a, ldc2=64, n_split=32),
                               None) == _lib.ERR_UNSUPPORTED  # n_split is no multiple of 256
    assert lib.b200_op_gemm_ex(None, None) == _lib.ERR_INVALID
