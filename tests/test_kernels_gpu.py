"""Each CUDA kernel alone against a plain PyTorch float32 reference of the same operation, at
sizes other than the engine's test models (widths and vocabularies that are no power of two,
head sizes in steps of 16, odd group counts)."""
import contextlib
import hashlib
import math

import pytest
import numpy as np
import torch

from plain import qwen2_plain as P

pytestmark = pytest.mark.gpu

DEV = "cuda:0"
DTYPES = [torch.float32, torch.bfloat16]


def K():
    from mini_hisparse_b200.kernels import api

    return api


def tol(dtype, scale=1.0):
    if dtype == torch.float32:
        return dict(atol=2e-5 * scale, rtol=2e-5)
    return dict(atol=1.6e-2 * scale, rtol=1.6e-2)


def rnd(*shape, dtype=torch.float32, seed=0, scale=1.0):
    g = torch.Generator().manual_seed(seed)
    return (torch.randn(*shape, generator=g) * scale).to(dtype).to(DEV)


# ---- embedding -----------------------------------------------------------------------------------
@pytest.mark.parametrize("dtype", DTYPES)
def test_embed(dtype):
    V, H = 777, 200
    table = rnd(V, H, dtype=dtype)
    tokens = torch.tensor([0, 776, 5, 5, 300], dtype=torch.int32, device=DEV)
    out = torch.empty(5, H, device=DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    K().embed(table, tokens, out, status)
    assert torch.equal(out, table.float()[tokens.long()]) and int(status) == 0
    bad = torch.tensor([3, 777, -1], dtype=torch.int32, device=DEV)
    out3 = torch.ones(3, H, device=DEV)
    K().embed(table, bad, out3, status)
    assert int(status) == 1 and torch.equal(out3[1:], torch.zeros(2, H, device=DEV))
    assert torch.equal(out3[0], table.float()[3])


@pytest.mark.parametrize("H", [4, 1028, 3584, 30])
@pytest.mark.parametrize("dtype", DTYPES)
def test_embed_forms(H, dtype):
    """Rows in steps of four elements and others, with a scale and a second copy, and an id outside the table."""
    table = rnd(50, H, dtype=dtype, seed=2)
    tokens = torch.tensor([3, 49, -1, 0], dtype=torch.int32, device=DEV)
    out, copy = torch.empty(4, H, device=DEV), torch.empty(4, H, dtype=torch.bfloat16, device=DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    K().embed(table, tokens, out, status, scale=1.5, copy=copy)
    want = table.float()[tokens.clamp(min=0).long()] * 1.5
    want[2] = 0
    assert int(status) == 1 and torch.equal(out, want) and torch.equal(copy, want.bfloat16())


# ---- RMSNorm ------------------------------------------------------------------------------------
@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("H", [80, 1000, 3584])
def test_rmsnorm_plain_add_rows_and_splits(dtype, H):
    R, eps = 7, 3e-6
    x = rnd(R, H, seed=1, scale=2.0)
    w = rnd(H, seed=2) * 0.1 + 1
    ref = P.rms_norm(x, w, eps)
    out = torch.empty(R, H, dtype=dtype, device=DEV)
    K().add_rmsnorm(x.clone(), w, eps, out)
    torch.testing.assert_close(out.float(), ref, **tol(dtype, 4))
    # with a delta: the residual is updated in place
    delta = rnd(R, H, dtype=dtype, seed=3)
    xr = x.clone()
    K().add_rmsnorm(xr, w, eps, out, delta=delta)
    torch.testing.assert_close(xr, x + delta.float(), atol=1e-6, rtol=1e-6)
    torch.testing.assert_close(out.float(), P.rms_norm(x + delta.float(), w, eps), **tol(dtype, 4))
    # split partials, summed in order
    parts = rnd(3, R, H, seed=4)
    xr = x.clone()
    K().add_rmsnorm(xr, w, eps, out, delta=parts, nsplit=3, split_stride=parts.stride(0))
    want = x + parts[0] + parts[1] + parts[2]
    torch.testing.assert_close(xr, want, atol=1e-6, rtol=1e-6)
    # selected rows: nothing is written back
    rows = torch.tensor([6, 0, 3], dtype=torch.int32, device=DEV)
    xr = x.clone()
    out3 = torch.empty(3, H, dtype=dtype, device=DEV)
    K().add_rmsnorm(xr, w, eps, out3, delta=delta, rows=rows)
    assert torch.equal(xr, x)
    torch.testing.assert_close(out3.float(), P.rms_norm((x + delta.float())[rows.long()], w, eps), **tol(dtype, 4))


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("R,H", [(512, 3584), (1531, 1000), (2048, 72), (700, 4096)])
def test_rmsnorm_many_rows(dtype, R, H):
    """The row-walking kernel of prompt portions (512 rows and more, rows of up to 4,096 elements): more rows
    than CTAs, a last round that not every CTA has, with and without a delta."""
    eps = 1e-5
    x = rnd(R, H, seed=1, scale=2.0)
    x[5] *= 40.0                                # one row far larger than the others: rows do not mix
    w = rnd(H, seed=2) * 0.1 + 1
    delta = rnd(R, H, dtype=dtype, seed=3)
    out = torch.full((R, H), float("nan"), dtype=dtype, device=DEV)
    xr = x.clone()
    K().add_rmsnorm(xr, w, eps, out, delta=delta)
    torch.testing.assert_close(xr, x + delta.float(), atol=1e-6, rtol=1e-6)
    torch.testing.assert_close(out.float(), P.rms_norm(x + delta.float(), w, eps), **tol(dtype, 4))
    out.fill_(float("nan"))
    xr = x.clone()
    K().add_rmsnorm(xr, w, eps, out)
    assert torch.equal(xr, x)
    torch.testing.assert_close(out.float(), P.rms_norm(x, w, eps), **tol(dtype, 4))


def test_residual_add():
    x = rnd(5, 33, seed=1)
    parts = rnd(2, 5, 33, seed=2)
    xr = x.clone()
    K().residual_add(xr, parts, nsplit=2, split_stride=parts.stride(0))
    torch.testing.assert_close(xr, x + parts[0] + parts[1], atol=1e-6, rtol=1e-6)


# ---- matrix product --------------------------------------------------------------------------------
@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("M,N,K_", [(1, 50, 24), (7, 1000, 96), (130, 67, 333), (65, 64, 16), (3, 129, 1)])
def test_gemm_simt(dtype, M, N, K_):
    a = rnd(M, K_, dtype=dtype, seed=1)
    w = rnd(N, K_, dtype=dtype, seed=2)
    bias = rnd(N, seed=3)
    ref = a.float() @ w.float().T
    out = torch.empty(M, N, dtype=torch.float32, device=DEV)
    K().gemm_simt(a, w, out)
    torch.testing.assert_close(out, ref, atol=2e-5 * math.sqrt(K_), rtol=2e-5)
    K().gemm_simt(a, w, out, bias=bias)
    torch.testing.assert_close(out, ref + bias, atol=2e-5 * math.sqrt(K_), rtol=2e-5)
    out_d = torch.empty(M, N, dtype=dtype, device=DEV)
    K().gemm_simt(a, w, out_d)
    torch.testing.assert_close(out_d.float(), ref, **tol(dtype, math.sqrt(K_)))
    parts = torch.full((3, M, N), float("nan"), device=DEV)
    K().gemm_simt(a, w, parts, nsplit=3, split_stride=parts.stride(0))
    torch.testing.assert_close(parts.sum(0), ref, atol=2e-5 * math.sqrt(K_), rtol=2e-5)


def test_gemm_is_true_float32():
    """A product that TF32 or bfloat16 inputs would get wrong by 1e-3 comes out to 1e-6."""
    a = torch.full((4, 64), 1.0 + 2 ** -12, device=DEV)
    w = torch.full((8, 64), 1.0 + 2 ** -12, device=DEV)
    out = torch.empty(4, 8, device=DEV)
    K().gemm_simt(a, w, out)
    exact = 64 * (1.0 + 2 ** -12) ** 2
    assert abs(float(out[0, 0]) - exact) < 1e-4


def float32_operands(kind, M, N, K_):
    """Operands of a float32 product: random ones, and ones that tell a kernel of fewer bits from one of 24."""
    a, w = rnd(M, K_, seed=1), rnd(N, K_, seed=2)
    if kind == "positive":
        a, w = a.abs(), w.abs()
    if kind == "one to two":
        a, w = 1 + a.abs().clamp(max=1), 1 + w.abs().clamp(max=1)
    if kind == "one number":                   # bits at the edge of every 8: cut from the top, parts 1, 2^-7 - 2^-15 and 2^-15 - 2^-23
        a, w = torch.full_like(a, 1 + 2.0 ** -7 - 2.0 ** -23), torch.full_like(w, 1 + 2.0 ** -7 - 2.0 ** -23)
    if kind == "tiny tokens":                  # their last bits are subnormal bfloat16 numbers, or below these
        a = a * 2.0 ** -118
    if kind == "tiny weights":
        w = w * 2.0 ** -118
    if kind == "huge":                         # parts and sums out of a scaled range
        a, w = a * 2.0 ** 113, w * 2.0 ** -20
    return a, w


@pytest.mark.parametrize("M", [1, 8, 9, 130])
@pytest.mark.parametrize("K_", [8, 16, 32, 40, 64, 104, 256, 3584])
@pytest.mark.parametrize("kind", ["signed", "positive", "one to two", "one number", "tiny tokens", "tiny weights", "huge"])
def test_float32_path_is_true_float32(M, K_, kind):
    """What the float32 path's products launch, on both sides of 8 tokens and of the shortest sum for the tensor cores, is no
    further from 64 bits than the chain of FFMA over K, in the largest error of an element and in the 2-norm."""
    from mini_hisparse_b200.kernels.runtime import Float32Runtime
    from mini_hisparse_b200.parts.base import Workspace

    N = 4096
    a, w = float32_operands(kind, M, N, K_)
    rt = Float32Runtime(DEV)
    rt.status = torch.zeros(1, dtype=torch.int32, device=DEV)
    p = rt.linear(a, w, Workspace(rt.device), "out")
    got = p.tensor.double().view(-1, M, N).sum(0)
    chain = torch.empty(M, N, device=DEV)
    K().gemm_simt(a, w, chain)
    ref = a.double() @ w.double().T
    assert int(rt.status) == 0 and got.isfinite().all()
    got, chain = (got - ref).abs(), (chain.double() - ref).abs()
    assert got.max() <= chain.max() and got.norm() <= chain.norm()


@pytest.mark.parametrize("M,N,K_,bn,nsplit", [
    (1, 5, 8, 0, 1), (2, 2400, 136, 0, 1), (3, 97, 1000, 0, 1), (4, 2369, 2056, 0, 1), (8, 130, 4104, 0, 1), (7, 2400, 520, 0, 1),
    (9, 130, 8, 64, 1), (64, 128, 32, 64, 1), (65, 127, 40, 64, 2), (33, 300, 1000, 64, 5), (128, 129, 96, 128, 1),
    (130, 128, 520, 128, 3), (97, 40, 2056, 128, 2), (192, 256, 64, 192, 1), (193, 130, 488, 192, 4), (400, 33, 3592, 192, 1),
])
@pytest.mark.parametrize("kind", ["signed", "positive", "special"])
def test_gemm_f32(M, N, K_, bn, nsplit, kind):
    """The float32 products at the edges of their tiles.  Bound, element by element, in units of 2^-24 S with S = sum |a||w|.
    Tensor cores: 1 for the parts' products that are left out; 2 for each of the two steps of a block of 32 that add products of
    first parts, of which a truncating sum of the block loses less than its last bit (2^-23), and less than 1 for the ten steps
    before them, which add at most 2^-7 as much; 1 per block for its rounded addition; 1 per split.  CUDA cores: 1 for every
    multiplication and addition of a lane (K / 32 of them at most), 5 across lanes, 8 across warps.  "special": infinities
    and NaN come out where a chain of multiplications and additions puts them."""
    a, w = rnd(M, K_, seed=1), rnd(N, K_, seed=2)
    if kind == "positive":
        a, w = a.abs(), w.abs()
    if kind == "special":
        a[M // 2, K_ // 2] = math.inf
        a[0, 0] = math.nan
        w[N - 1, K_ // 2] = -math.inf
        a[M - 1, K_ - 1] = 3.4e38          # rounded to 8 bits it is infinite
        w[:, K_ - 1] = 2.0 ** -20          # ... and none of its products overflows, which 64 bits would not show
    out = torch.full((nsplit, M, N), math.nan, device=DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    parts = torch.empty(3 * M * K_, dtype=torch.bfloat16, device=DEV) if bn else None
    K().gemm_f32(a, w, out, bn=bn, nsplit=nsplit, split_stride=out.stride(0), parts=parts, status=status)
    got, ref = out.double().sum(0), a.double() @ w.double().T
    assert int(status) == 0
    if kind == "special":
        ref = ref.float().double()
        assert torch.equal(got.isnan(), ref.isnan()) and torch.equal(got[got.isinf()], ref[ref.isinf()])
    room = (6 + -(-K_ // 32) + nsplit if bn else -(-K_ // 32) + 4 + 5 + 8) * 2.0 ** -24 * (a.abs().double() @ w.abs().double().T)
    fine = ref.isfinite()
    assert ((got - ref).abs() <= room)[fine].all()


@pytest.mark.parametrize("M,I,K_", [(1, 3, 40), (2, 256, 96), (4, 256, 96), (3, 1183, 3584), (5, 1185, 200), (8, 4000, 1024), (7, 33, 4096)])
def test_gemm_f32_gate_in_the_product(M, I, K_):
    """silu(x Wg^T) * (x Wu^T) of few tokens in one kernel, two and four features a warp, K shared by warps or not, against 64
    bits: each sum within its bound, carried through the gate (whose slope is below 1.1)."""
    x, w = rnd(M, K_, seed=1), rnd(2 * I, K_, seed=2, scale=K_ ** -0.5)
    out = torch.full((M + 1, I), float("nan"), device=DEV)
    K().gemm_f32_glu(x, w, out[:M])
    g, u = (x.double() @ w.double().T).split(I, 1)
    eg, eu = ((-(-K_ // 32) + 17) * 2.0 ** -24 * (x.abs().double() @ w.abs().double().T)).split(I, 1)
    room = 1.1 * eg * u.abs() + g.abs() * eu + 8 * 2.0 ** -24 * (g * u).abs() + 1e-30
    assert bool(out[M].isnan().all()) and ((out[:M].double() - torch.nn.functional.silu(g) * u).abs() <= room).all()
    with pytest.raises(Exception, match="gemm_f32_glu"):
        K().gemm_f32_glu(rnd(9, K_, seed=1), w, torch.empty(9, I, device=DEV))


def test_gemm_f32_takes():
    """What the float32 kernels do not take is refused by the entry point and known beforehand."""
    a, w = rnd(20, 64, seed=1), rnd(30, 64, seed=2)
    assert K().gemm_f32_takes(a, w)
    assert not K().gemm_f32_takes(a[:, :60], w[:, :60])           # K in steps of 8
    assert not K().gemm_f32_takes(a[:, 1:57], w[:, :56])          # rows off 16 bytes
    assert not K().gemm_f32_takes(a.bfloat16(), w)
    out = torch.empty(20, 30, device=DEV)
    for bad in (dict(), dict(bn=64), dict(bn=100, parts=torch.empty(3 * 20 * 64, dtype=torch.bfloat16, device=DEV))):
        with pytest.raises(Exception, match="gemm_f32"):
            K().gemm_f32(a, w, out, **bad)


@pytest.mark.parametrize("M,N,K_,swap,bn,nsplit", [
    (128, 128, 64, False, 128, 1), (200, 300, 136, False, 128, 1), (333, 1000, 3584, False, 256, 1),
    (70, 520, 200, False, 128, 2), (8, 256, 512, True, 16, 1), (1, 777, 96, True, 16, 1),
    (17, 1000, 3584, True, 32, 7), (64, 130, 1024, True, 64, 4), (2048, 2000, 512, False, 256, 1),
])
@pytest.mark.parametrize("out_dtype", DTYPES)
def test_gemm_tensor_core(M, N, K_, swap, bn, nsplit, out_dtype):
    """The tcgen05 product against float32 matmul of the same bfloat16 values: ragged edges in
    every dimension, both operand orders, split K."""
    a = rnd(M, K_, dtype=torch.bfloat16, seed=1)
    w = rnd(N, K_, dtype=torch.bfloat16, seed=2)
    ref = a.float() @ w.float().T
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    if nsplit > 1:
        if out_dtype != torch.float32:
            pytest.skip("partials are float32")
        out = torch.full((nsplit, M, N), float("nan"), device=DEV)
        K().gemm_tc(a, w, out, swap=swap, bn=bn, nsplit=nsplit, split_stride=out.stride(0), status=status)
        got = out.sum(0)
    else:
        out = torch.full((M + 1, N), float("nan"), dtype=out_dtype, device=DEV)
        K().gemm_tc(a, w, out[:M], swap=swap, bn=bn, status=status)
        assert bool(out[M].isnan().all())               # nothing written past the last row
        got = out[:M].float()
    assert int(status) == 0
    if out_dtype == torch.float32:
        torch.testing.assert_close(got, ref, atol=3e-5 * math.sqrt(K_) * 4, rtol=2e-5)
    else:
        torch.testing.assert_close(got, ref, atol=1e-2 * float(ref.abs().max()), rtol=1e-2)


@pytest.mark.parametrize("M,N,K_", [(65, 64, 64), (128, 128, 64), (200, 300, 136), (333, 1000, 3584), (100, 7168, 1024),
                                    (2048, 2000, 512), (1024, 520, 13824), (700, 4608, 3584), (129, 40, 8192),
                                    (2048, 2600, 8192), (1100, 5000, 8256), (2300, 2304, 8960)])
@pytest.mark.parametrize("shared", [True, False])
@pytest.mark.parametrize("out_dtype", DTYPES)
def test_gemm_persistent(M, N, K_, shared, out_dtype):
    """The persistent product: ragged edges, fewer tiles than SMs, and (the last three shapes: a
    long K and a last round that fills a part of the SMs) CTAs that share tiles' K ranges through
    the workspace; the same shapes without a workspace.  Twice in a row: the flags are left zero."""
    a = rnd(M, K_, dtype=torch.bfloat16, seed=1)
    w = rnd(N, K_, dtype=torch.bfloat16, seed=2)
    ref = a.float() @ w.float().T
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    scratch = K().stream_k_scratch(DEV) if shared else None
    outs = []
    for _ in range(2):
        out = torch.full((M + 1, N), float("nan"), dtype=out_dtype, device=DEV)
        K().gemm_tc(a, w, out[:M], swap=False, bn=0, status=status, scratch=scratch)
        assert bool(out[M].isnan().all())
        outs.append(out[:M].float())
    assert int(status) == 0
    if shared:
        assert int(scratch[1].abs().sum()) == 0
    assert torch.equal(outs[0], outs[1])                 # the order of the sums is fixed
    if out_dtype == torch.float32:
        torch.testing.assert_close(outs[0], ref, atol=3e-5 * math.sqrt(K_) * 4, rtol=2e-5)
    else:
        torch.testing.assert_close(outs[0], ref, atol=1e-2 * float(ref.abs().max()), rtol=1e-2)


def test_gemm_persistent_wait_that_runs_out_is_reported_and_the_kernel_stays_usable():
    """A bounded wait made to run out by a flag that nothing sets: the counters through which the CTAs
    that share a tile's K range meet are preset so that their count is never reached.  With a short
    limit the CTAs give up within milliseconds: status bit 4 is set, the kernel returns (its MMAs
    drained, its copies landed, its tensor memory freed), and after the flags are put back to zero
    (what the runner does after such an error) the same product is right again."""
    M, N, K_ = 2300, 2304, 8960                       # its last round of tiles is shared eight ways along K
    a = rnd(M, K_, dtype=torch.bfloat16, seed=1)
    w = rnd(N, K_, dtype=torch.bfloat16, seed=2)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    scratch = K().stream_k_scratch(DEV)
    out = torch.zeros(M, N, dtype=torch.bfloat16, device=DEV)
    scratch[1].fill_(-1000)
    with K().gemm_tc_wait_limit(2000):
        K().gemm_tc(a, w, out, swap=False, bn=0, status=status, scratch=scratch)
        torch.cuda.synchronize()
    assert int(status) & 4
    from mini_hisparse_b200.engine.step import ModelRunner
    assert "tensor-core matrix product" in ModelRunner.status_message(int(status))
    status.zero_()
    scratch[1].zero_()
    K().gemm_tc(a, w, out, swap=False, bn=0, status=status, scratch=scratch)
    assert int(status) == 0 and int(scratch[1].abs().sum()) == 0
    ref = a.float() @ w.float().T
    torch.testing.assert_close(out.float(), ref, atol=1e-2 * float(ref.abs().max()), rtol=1e-2)


@pytest.mark.parametrize("M,I,K_,swap,bn", [(200, 176, 64, False, 256), (2048, 1184, 512, False, 256),
                                              (200, 176, 64, False, 0), (2048, 1184, 512, False, 0), (130, 2000, 3584, False, 0),
                                              (2048, 1312, 8192, False, 0),
                                              (8, 176, 96, True, 16), (33, 304, 3584, True, 64), (1, 18944, 128, True, 16)])
def test_gemm_tensor_core_swiglu_epilogue(M, I, K_, swap, bn):
    """silu(x Wg^T) * (x Wu^T) written by the product's epilogue from block-interleaved weights."""
    x = rnd(M, K_, dtype=torch.bfloat16, seed=1)
    gate = rnd(I, K_, dtype=torch.bfloat16, seed=2, scale=0.2)
    up = rnd(I, K_, dtype=torch.bfloat16, seed=3, scale=0.2)
    w = torch.stack((gate.view(I // 16, 16, K_), up.view(I // 16, 16, K_)), 1).reshape(2 * I, K_).contiguous()
    out = torch.full((M + 1, I), float("nan"), dtype=torch.bfloat16, device=DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    K().gemm_tc_swiglu(x, w, out[:M], swap=swap, bn=bn, status=status,
                       scratch=K().stream_k_scratch(DEV) if bn == 0 else None)
    g, u = x.float() @ gate.float().T, x.float() @ up.float().T
    ref = g * torch.sigmoid(g) * u
    assert int(status) == 0 and bool(out[M].isnan().all())
    torch.testing.assert_close(out[:M].float(), ref, atol=1e-2 * float(ref.abs().max()), rtol=1.6e-2)
    # the stand-alone gate kernel reads the same interleaved layout
    gu = (x.float() @ w.float().T).to(torch.bfloat16)
    out2 = torch.empty(M, I, dtype=torch.bfloat16, device=DEV)
    K().swiglu(gu, out2, block=16)
    torch.testing.assert_close(out2.float(), ref, atol=2e-2 * float(ref.abs().max()), rtol=2e-2)


@pytest.mark.parametrize("M,N,K_", [(257, 19000, 136), (272, 27648, 64), (543, 27648, 200), (543, 7168, 1024), (321, 14001, 72),
                                    (781, 13826, 64)])
@pytest.mark.parametrize("epilogue", ["float32", "bfloat16", "silu", "gelu_tanh", "gelu_act", "heads128", "heads64"])
def test_gemm_tiles_of_features(M, N, K_, epilogue):
    """Token counts that fill tiles of 256 tokens badly: the two-SM kernel with 256 features a tile and every epilogue,
    ragged in tokens and features, output rows on and off 16 bytes."""
    x = rnd(M, K_, dtype=torch.bfloat16, seed=1)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    scratch = K().stream_k_scratch(DEV)
    if epilogue.startswith("heads"):
        d = int(epilogue[5:])
        nkv, P_ = 3, 16
        nq = N // d - 2 * nkv
        n = (nq + 2 * nkv) * d
        w, bias = rnd(n, K_, dtype=torch.bfloat16, seed=2, scale=K_ ** -0.5), rnd(n, seed=3)
        pos = torch.arange(5, 5 + M, dtype=torch.int32, device=DEV)
        seg = torch.zeros(M, dtype=torch.int32, device=DEV)
        pages = (M + 5) // P_ + 1
        table = torch.randperm(pages, generator=torch.Generator().manual_seed(5)).to(torch.int32).to(DEV)[None]
        inv = (10000.0 ** (-torch.arange(0, d, 2).float() / d)).to(DEV)
        for rdim, interleaved in ((d, False), (d // 2, True)):
            cs = torch.empty(M, rdim, device=DEV)
            K().rope_table(pos, inv[: rdim // 2], cs)
            q, cache = torch.full((M + 1, nq * d), float("nan"), dtype=torch.bfloat16, device=DEV), torch.zeros(pages, 2, nkv, P_, d, dtype=torch.bfloat16, device=DEV)
            K().gemm_tc_qkv_rope(x, w, bias, cs, pos, seg, table, q[:M], cache, nq=nq, nkv=nkv, d=d, page_size=P_, rotary_dim=rdim,
                                 interleaved=interleaved, status=status)
            y = (x.float() @ w.float().T + bias).view(M, -1, d)
            h, c, s = rdim // 2, cs[:, None, : rdim // 2], cs[:, None, rdim // 2:]
            a, b = (y[..., 0:rdim:2], y[..., 1:rdim:2]) if interleaved else (y[..., :h], y[..., h:rdim])
            turned = torch.stack((a * c - b * s, b * c + a * s), -1).flatten(-2) if interleaved else torch.cat((a * c - b * s, b * c + a * s), -1)
            y = torch.cat((torch.cat((turned, y[..., rdim:]), -1)[:, : nq + nkv], y[:, nq + nkv:]), 1)
            page, at = table[0][(pos // P_).long()].long(), (pos % P_).long()
            top = float(y.abs().max())
            assert int(status) == 0 and bool(q[M].isnan().all())
            torch.testing.assert_close(q[:M].float(), y[:, :nq].flatten(1), atol=2.0 ** -8 * top, rtol=2.0 ** -8)
            for plane in (0, 1):
                got = cache[page, plane, :, at].float()
                torch.testing.assert_close(got, y[:, nq + plane * nkv: nq + (plane + 1) * nkv], atol=2.0 ** -8 * top, rtol=2.0 ** -8)
            assert int((cache[:, 0].abs().sum(-1) > 0).sum()) == M * nkv
        return
    gated = epilogue in ("silu", "gelu_tanh")
    n = N // 32 * 32 if gated else N
    w = rnd(n, K_, dtype=torch.bfloat16, seed=2, scale=0.2)
    out = torch.full((M + 1, n // 2 if gated else n), float("nan"), dtype=torch.float32 if epilogue == "float32" else torch.bfloat16, device=DEV)
    y = x.float() @ w.float().T
    if gated:
        K().gemm_tc_glu(x, w, out[:M], epilogue, swap=False, bn=0, status=status, scratch=scratch)
        g, u = y.view(M, -1, 2, 16).unbind(2)
        y = ((torch.nn.functional.silu(g) if epilogue == "silu" else torch.nn.functional.gelu(g, approximate="tanh")) * u).flatten(1)
    elif epilogue == "gelu_act":
        K().gemm_tc_act(x, w, out[:M], "gelu_tanh", status=status, scratch=scratch)
        y = torch.nn.functional.gelu(y, approximate="tanh")
    else:
        K().gemm_tc(x, w, out[:M], swap=False, bn=0, status=status, scratch=scratch)
    assert int(status) == 0 and bool(out[M].isnan().all())
    if epilogue == "float32":       # two float32 sums of K exact products
        torch.testing.assert_close(out[:M], y, atol=2.0 * K_ * 2.0 ** -24 * float((x.float().abs() @ w.float().abs().T).max()), rtol=0)
    else:
        torch.testing.assert_close(out[:M].float(), y, atol=2.0 ** -8 * float(y.abs().max()), rtol=2.0 ** -8)


@pytest.mark.parametrize("M,N,K_", [(543, 14001, 2056), (272, 13826, 2056), (543, 27650, 3080), (321, 27648, 3080)])
@pytest.mark.parametrize("epilogue", ["float32", "bfloat16", "silu", "gelu_tanh", "gelu_act", "heads128", "heads64"])
def test_gemm_tiles_of_features_where_they_are_taken(M, N, K_, epilogue):
    """The same at sizes of which the choice (made for whole products' times) takes this form with every epilogue."""
    from ctypes import c_int

    from mini_hisparse_b200.kernels import build

    kind, step = {"silu": (1, 32), "gelu_tanh": (3, 32), "gelu_act": (4, 1), "heads128": (2, 128), "heads64": (2, 64)}.get(epilogue, (0, 1))
    pairs = torch.cuda.get_device_properties(0).multi_processor_count // 2
    if pairs == 74:
        assert build.load("gemm_tc").mhb_gemm_tc_pair_form(c_int(M), c_int(N // step * step), c_int(K_), c_int(pairs), c_int(kind)) > 0
    test_gemm_tiles_of_features(M, N, K_, epilogue)


@pytest.mark.parametrize("T,I,block,nsplit", [(1, 4, 4, 1), (3, 1020, 1020, 1), (5, 1028, 4, 3), (562, 304, 16, 1), (2, 176, 16, 9), (7, 102, 102, 2),
                                              (3, 30, 6, 1)])
@pytest.mark.parametrize("dtype", DTYPES)
def test_swiglu_four_at_a_time(T, I, block, nsplit, dtype):
    """silu(gate) * up in both layouts, in widths that are taken four elements at a time and widths that are not, from parts."""
    parts = rnd(nsplit, T, 2 * I, seed=T + I)
    out = torch.full((T + 1, I), float("nan"), dtype=dtype, device=DEV)
    K().swiglu(parts if nsplit > 1 else parts[0], out[:T], nsplit=nsplit, split_stride=parts.stride(0), block=block)
    g, u = parts.double().sum(0).view(T, -1, 2, block).unbind(2)
    ref = (torch.nn.functional.silu(g) * u).reshape(T, I)
    assert bool(out[T].isnan().all())
    torch.testing.assert_close(out[:T].double(), ref, atol=1e-5, rtol=2.0 ** -8 if dtype == torch.bfloat16 else 1e-5)


def test_gemm_tensor_core_refuses_unaligned_k():
    from mini_hisparse_b200.kernels.api import KernelError

    a = rnd(4, 100, dtype=torch.bfloat16)
    w = rnd(9, 100, dtype=torch.bfloat16)
    with pytest.raises(KernelError, match="multiples of 8"):
        K().gemm_tc(a, w, torch.empty(4, 9, device=DEV), swap=True, bn=16)


@pytest.mark.parametrize("nq,nkv,d,P_,T,Kd", [(28, 4, 128, 16, 300, 3584), (3, 1, 64, 32, 70, 192), (5, 5, 128, 8, 129, 256),
                                               (2, 1, 64, 16, 2100, 64)])
@pytest.mark.parametrize("rdim_of,interleaved", [(lambda d: d, False), (lambda d: 0, False), (lambda d: d, True),
                                                 (lambda d: d // 2, False), (lambda d: d // 4 * 3, True)],
                         ids=["half_split", "none", "interleaved", "partial_half_split", "partial_interleaved"])
def test_gemm_qkv_epilogue_rotates_and_appends(nq, nkv, d, P_, T, Kd, rdim_of, interleaved):
    """The q/k/v product whose epilogue adds the bias, rotates and appends to the paged cache,
    against the product followed by the rotary kernel (which has its own test against the plain
    formulas): two segments, one of which starts inside a page; every rotation style."""
    rdim = rdim_of(d)
    assert K().gemm_tc_qkv_rope_supports(d, rdim, interleaved)
    N = (nq + 2 * nkv) * d
    x = rnd(T, Kd, dtype=torch.bfloat16, seed=1)
    w = rnd(N, Kd, dtype=torch.bfloat16, seed=2, scale=1.0 / math.sqrt(Kd))
    bias = rnd(N, seed=3) * 0.1
    theta = 10000.0
    inv = (theta ** (-torch.arange(0, rdim, 2).float() / rdim)).to(DEV) if rdim else None
    n0 = T // 3
    positions = torch.tensor(list(range(37, 37 + n0)) + list(range(0, T - n0)), dtype=torch.int32, device=DEV)
    tok_seg = torch.tensor([0] * n0 + [1] * (T - n0), dtype=torch.int32, device=DEV)
    pages0, pages1 = -(-(37 + n0) // P_), -(-(T - n0) // P_)
    num_pages = pages0 + pages1 + 3
    perm = torch.randperm(num_pages, generator=torch.Generator().manual_seed(5)).tolist()
    table = torch.full((2, max(pages0, pages1)), -1, dtype=torch.int32)
    table[0, :pages0] = torch.tensor(perm[:pages0])
    table[1, :pages1] = torch.tensor(perm[pages0:pages0 + pages1])
    table = table.to(DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    # reference: float32 product, then the rotary kernel
    qkv = torch.empty(T, N, device=DEV)
    K().gemm_simt(x.float(), w.float(), qkv)
    q_ref = torch.empty(T, nq * d, dtype=torch.bfloat16, device=DEV)
    cache_ref = torch.zeros(num_pages, 2, nkv, P_, d, dtype=torch.bfloat16, device=DEV)
    K().rope_append(qkv, bias, positions, tok_seg, table, inv, q_ref, cache_ref, nq=nq, nkv=nkv, d=d, page_size=P_,
                    rotary_dim=rdim, interleaved=interleaved, status=status)
    cs = None
    if rdim:
        cs = torch.empty(T, rdim, device=DEV)
        K().rope_table(positions, inv, cs)
    q = torch.full((T, nq * d), float("nan"), dtype=torch.bfloat16, device=DEV)
    cache = torch.zeros(num_pages, 2, nkv, P_, d, dtype=torch.bfloat16, device=DEV)
    K().gemm_tc_qkv_rope(x, w, bias, cs, positions, tok_seg, table, q, cache, nq=nq, nkv=nkv, d=d, page_size=P_,
                         rotary_dim=rdim, interleaved=interleaved, status=status)
    assert int(status) == 0
    scale = float(qkv.abs().max())
    torch.testing.assert_close(q.float(), q_ref.float(), atol=1e-2 * scale, rtol=1.6e-2)
    torch.testing.assert_close(cache.float(), cache_ref.float(), atol=1e-2 * scale, rtol=1.6e-2)
    written, written_ref = cache.abs().sum(-1) > 0, cache_ref.abs().sum(-1) > 0          # per (page, plane, head, slot)
    assert bool(written_ref.any()) and bool((written == written_ref).all())            # the same slots were written
    # without write access nothing is appended
    cache2 = torch.zeros_like(cache)
    K().gemm_tc_qkv_rope(x, w, bias, cs, positions, tok_seg, table, q, cache2, nq=nq, nkv=nkv, d=d, page_size=P_,
                         rotary_dim=rdim, interleaved=interleaved, write_kv=False, status=status)
    assert int(cache2.abs().sum()) == 0


# ---- rotary + append -----------------------------------------------------------------------------
def plain_rotation(t, positions, theta, rdim, interleaved):
    """The first rdim elements of every head of t [T, heads, d] turned by angle_i = pos * theta^(-2i/rdim):
    pairs (i, i + rdim/2), or (2i, 2i + 1) if interleaved; the rest of the head passes.  With rdim = d
    and half-split pairs this is the reference's rotation (mini_hisparse/model.py:141-151)."""
    if rdim == 0:
        return t
    inv = theta ** (-torch.arange(0, rdim, 2, device=t.device).float() / rdim)
    ang = positions.float()[:, None] * inv[None, :]
    cos, sin = ang.cos()[:, None, :], ang.sin()[:, None, :]
    out = t.clone()
    if interleaved:
        a, b = t[..., 0:rdim:2], t[..., 1:rdim:2]
        out[..., 0:rdim:2], out[..., 1:rdim:2] = a * cos - b * sin, b * cos + a * sin
    else:
        a, b = t[..., : rdim // 2], t[..., rdim // 2: rdim]
        out[..., : rdim // 2], out[..., rdim // 2: rdim] = a * cos - b * sin, b * cos + a * sin
    return out


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("nq,nkv,d,P_,rdim,interleaved", [
    (4, 2, 16, 16, 16, False), (3, 1, 32, 32, 32, False), (10, 2, 48, 16, 48, False), (7, 7, 128, 8, 128, False),
    (3, 1, 32, 24, 32, True), (10, 2, 48, 7, 24, False), (2, 2, 64, 16, 40, True), (5, 1, 80, 16, 6, True),
    (2, 1, 18, 16, 10, False), (4, 4, 64, 16, 0, False)])
def test_rope_append(dtype, nq, nkv, d, P_, rdim, interleaved):
    """Every rotation style against the plain rotation: the reference's (half-split pairs over the
    whole head), interleaved pairs, a rotated part of the head (widths that the vector kernel takes and
    widths that only the scalar kernel takes), and none."""
    theta = 50000.0
    T, pages = 21, 9
    width = (nq + 2 * nkv) * d
    qkv = rnd(T, width, seed=1)
    bias = rnd(width, seed=2) * 0.1
    # two segments: one starts at position 37 (inside a page), one at 0
    positions = torch.tensor(list(range(37, 37 + 13)) + list(range(0, 8)), dtype=torch.int32, device=DEV)
    tok_seg = torch.tensor([0] * 13 + [1] * 8, dtype=torch.int32, device=DEV)
    w_pages = -(-(37 + 13) // P_)
    table = torch.full((2, max(w_pages, 2)), -1, dtype=torch.int32)
    perm = torch.randperm(64, generator=torch.Generator().manual_seed(5)).tolist()
    table[0, :w_pages] = torch.tensor(perm[:w_pages])
    table[1, : -(-8 // P_)] = torch.tensor(perm[w_pages : w_pages + -(-8 // P_)])
    table = table.to(DEV)
    cache = torch.zeros(64, 2, nkv, P_, d, dtype=dtype, device=DEV)
    q_out = torch.empty(T, nq * d, dtype=dtype, device=DEV)
    inv = (theta ** (-torch.arange(0, rdim, 2).float() / rdim)).to(DEV) if rdim else None
    K().rope_append(qkv, bias, positions, tok_seg, table, inv, q_out, cache, nq=nq, nkv=nkv, d=d, page_size=P_,
                    rotary_dim=rdim, interleaved=interleaved)
    full = qkv + bias
    q = full[:, : nq * d].view(T, nq, d)
    k = full[:, nq * d : (nq + nkv) * d].view(T, nkv, d)
    v = full[:, (nq + nkv) * d :].view(T, nkv, d)
    if rdim == d and not interleaved:          # the reference's own form, as the plain model computes it
        cos, sin = P.rope_tables(positions, d, theta, torch.float32)
        torch.testing.assert_close(plain_rotation(q, positions, theta, rdim, False), P.rotate(q, cos, sin),
                                   atol=1e-5, rtol=1e-5)
    torch.testing.assert_close(q_out.float().view(T, nq, d), plain_rotation(q, positions, theta, rdim, interleaved),
                               **tol(dtype, 4))
    kr = plain_rotation(k, positions, theta, rdim, interleaved)
    for t in range(T):
        pos, seg = int(positions[t]), int(tok_seg[t])
        page = int(table[seg, pos // P_])
        torch.testing.assert_close(cache[page, 0, :, pos % P_].float(), kr[t], **tol(dtype, 4))
        torch.testing.assert_close(cache[page, 1, :, pos % P_].float(), v[t], **tol(dtype, 4))
    # nothing else was touched
    touched = torch.zeros(64, P_, dtype=torch.bool)
    for t in range(T):
        pos, seg = int(positions[t]), int(tok_seg[t])
        touched[int(table[seg, pos // P_]), pos % P_] = True
    untouched = cache.float().abs().sum((1, 2, 4)).cpu()[~touched]
    assert float(untouched.sum()) == 0.0


def test_rope_append_refuses_a_page_outside_the_pool():
    nq, nkv, d, P_ = 2, 1, 16, 16
    qkv = rnd(1, 4 * d)
    pos = torch.tensor([3], dtype=torch.int32, device=DEV)
    seg = torch.zeros(1, dtype=torch.int32, device=DEV)
    table = torch.tensor([[99]], dtype=torch.int32, device=DEV)
    cache = torch.zeros(4, 2, nkv, P_, d, device=DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    inv = torch.ones(d // 2, device=DEV)
    q_out = torch.empty(1, nq * d, device=DEV)
    K().rope_append(qkv, None, pos, seg, table, inv, q_out, cache, nq=nq, nkv=nkv, d=d, page_size=P_, status=status)
    assert int(status) == 2 and float(cache.abs().sum()) == 0.0


# ---- SwiGLU -------------------------------------------------------------------------------------
@pytest.mark.parametrize("dtype", DTYPES)
def test_swiglu(dtype):
    T, I = 5, 176
    gu = rnd(T, 2 * I, dtype=dtype, seed=1, scale=3)
    out = torch.empty(T, I, dtype=dtype, device=DEV)
    K().swiglu(gu, out)
    g, u = gu.float()[:, :I], gu.float()[:, I:]
    torch.testing.assert_close(out.float(), g * torch.sigmoid(g) * u, **tol(dtype, 8))
    parts = rnd(2, T, 2 * I, seed=2)
    K().swiglu(parts, out, nsplit=2, split_stride=parts.stride(0))
    s = parts.sum(0)
    torch.testing.assert_close(out.float(), s[:, :I] * torch.sigmoid(s[:, :I]) * s[:, I:], **tol(dtype, 8))


# ---- attention -------------------------------------------------------------------------------------
def paged_case(nq, nkv, d, P_, seg_specs, dtype, seed=0):
    """Segments (history, new tokens): K/V of the history AND the new tokens are in shuffled pages
    (the engine appends before it attends)."""
    from mini_hisparse_b200.parts.base import Segment

    pool = sum(-(-(h + n) // P_) for h, n in seg_specs) + 13
    g = torch.Generator().manual_seed(seed)
    perm = torch.randperm(pool, generator=g).tolist()
    cache = torch.zeros(pool, 2, nkv, P_, d, dtype=dtype, device=DEV)
    cache.normal_(generator=torch.Generator(device=DEV).manual_seed(seed))   # stale junk everywhere
    segments, ks, vs, qs, positions = [], [], [], [], []
    width = max(-(-(h + n) // P_) for h, n in seg_specs)
    table = torch.full((len(seg_specs), width), -1, dtype=torch.int32)
    off = 0
    for si, (hist, n) in enumerate(seg_specs):
        total = hist + n
        k = torch.randn(total, nkv, d, generator=g).to(dtype)
        v = torch.randn(total, nkv, d, generator=g).to(dtype)
        q = torch.randn(total, nq, d, generator=g).to(dtype)
        npg = -(-total // P_)
        pages = [perm.pop() for _ in range(npg)]
        table[si, :npg] = torch.tensor(pages)
        for t in range(total):
            cache[pages[t // P_], 0, :, t % P_] = k[t].to(DEV)
            cache[pages[t // P_], 1, :, t % P_] = v[t].to(DEV)
        segments.append(Segment(si, si, hist, n, off))
        ks.append(k), vs.append(v), qs.append(q)
        positions += list(range(hist, total))
        off += n
    return cache, table.to(DEV), segments, qs, ks, vs, torch.tensor(positions, dtype=torch.int32, device=DEV)


def run_attention(nq, nkv, d, P_, seg_specs, dtype, window=None, fixed_nsplit=None, seed=0, edit=None,
                  kernel="simt"):
    from mini_hisparse_b200.parts.attention import ITEM_INTS, AttentionShape, plan_attention

    cache, table, segments, qs, ks, vs, positions = paged_case(nq, nkv, d, P_, seg_specs, dtype, seed)
    if edit:
        edit(qs, ks, vs, cache, table)
    T = sum(n for _, n in seg_specs)
    need = AttentionShape(nq, nkv, window, {"mma": 64, "tc": 128}.get(kernel, 16))
    plan = plan_attention(need, segments, T, 148, fixed_nsplit=fixed_nsplit)
    q = torch.cat([qq[h:] for qq, (h, n) in zip(qs, seg_specs)]).reshape(T, nq * d).to(DEV)
    out = torch.full((T, nq * d), float("nan"), dtype=dtype, device=DEV)
    rows = max(1, plan.part_rows)
    part_acc = torch.full((rows, nq, d), float("nan"), device=DEV)
    part_ml = torch.full((rows, nq, 2), float("nan"), device=DEV)
    items = torch.from_numpy(plan.items).to(DEV).reshape(-1)
    tpr = torch.from_numpy(plan.tok_part_row).to(DEV)
    tns = torch.from_numpy(plan.tok_nsplit).to(DEV)
    n_items = plan.items.shape[0]
    kw = dict(nq=nq, nkv=nkv, d=d, page_size=P_, window=window or 0)
    # "tc": short segments by the TMA-fed mma kernel, long portions by the tcgen05 kernel (the engine's pairing)
    fused = kernel in ("mma", "tc") and seed % 2 == 0     # the kernel merges its own key splits
    if kernel in ("mma", "tc"):
        launch = K().attention_mma if kernel == "mma" else K().attention_tma
        if plan.n_small:
            groups = nq // nkv
            counters = torch.zeros(T * nkv * -(-groups // 16), dtype=torch.int32, device=DEV) if fused else None
            launch(q, cache, out, part_acc, part_ml, items, plan.n_small, 16, positions, table, tpr,
                   tok_nsplit=tns, counters=counters, **kw)
            if fused:
                assert int(counters.abs().sum()) == 0        # left zero for the next launch
        if plan.n_big and kernel == "tc":
            status = torch.zeros(1, dtype=torch.int32, device=DEV)
            K().attention_tc(q, cache, out, items[plan.n_small * ITEM_INTS:], plan.n_big, positions, table,
                             status=status, part_acc=part_acc, part_ml=part_ml, tok_part_row=tpr, **kw)
            assert int(status) == 0
            if plan.big_split:                               # long tiles were split along the keys
                K().attention_combine(part_acc, part_ml, tpr, tns, out, nq=nq, d=d)
        elif plan.n_big:
            launch(q, cache, out, part_acc, part_ml, items[plan.n_small * ITEM_INTS:], plan.n_big, 64,
                   positions, table, tpr, **kw)
    else:
        K().attention_simt(q, cache, out, part_acc, part_ml, items, n_items, n_items, positions, table, tpr, **kw)
    if plan.part_rows and not fused:
        K().attention_combine(part_acc, part_ml, tpr, tns, out, nq=nq, d=d)
    ref = torch.cat([
        P.causal_attention(qq.float(), kk.float(), vv.float(), window=window)[h:]
        for qq, kk, vv, (h, n) in zip(qs, ks, vs, seg_specs)
    ]).reshape(T, nq * d)
    return out.float().cpu(), ref, plan


@pytest.mark.parametrize("nq,nkv,d,P_", [(3, 1, 32, 32), (28, 4, 128, 16), (16, 4, 64, 5), (8, 1, 100, 7), (5, 5, 4, 1), (70, 1, 8, 16)])
@pytest.mark.parametrize("window", [None, 70])
@pytest.mark.parametrize("dtype", DTYPES)
def test_attention_rows(nq, nkv, d, P_, window, dtype):
    """Prompt portions on the CUDA cores in tiles of 64 query rows: portions behind a history and at the start, ragged tiles,
    keys around a tile of 32, more heads per KV head than a tile has rows, against 64 bits."""
    from mini_hisparse_b200.parts.attention import AttentionShape, plan_attention

    specs = [(0, 17), (0, 33), (31, 40), (64, 64), (100, 65), (5, 90)]
    cache, table, segments, qs, ks, vs, positions = paged_case(nq, nkv, d, P_, specs, dtype)
    T = sum(n for _, n in specs)
    plan = plan_attention(AttentionShape(nq, nkv, window, 64, cuda_cores=True), segments, T, 148)
    assert plan.n_small == 0 and plan.n_big and not plan.big_split
    q = torch.cat([qq[h:] for qq, (h, n) in zip(qs, specs)]).reshape(T, nq * d).to(DEV)
    out = torch.full((T + 1, nq * d), float("nan"), dtype=dtype, device=DEV)
    K().attention_rows(q, cache, out[:T], torch.from_numpy(plan.items).to(DEV).reshape(-1), plan.n_big, positions, table, nq=nq, nkv=nkv,
                       d=d, page_size=P_, window=window or 0)
    ref = []
    for qq, kk, vv, (h, n) in zip(qs, ks, vs, specs):
        qq, kk, vv = (y.to(dtype).double() for y in (qq, kk, vv))
        kk, vv = (y.repeat_interleave(nq // nkv, 1) for y in (kk, vv))
        z = torch.einsum("qhd,khd->hqk", qq[h:], kk) * d ** -0.5
        far = torch.arange(h, h + n)[:, None] - torch.arange(h + n)
        z.masked_fill_((far < 0) | (far >= (window or 1 << 30)), -math.inf)
        ref.append(torch.einsum("hqk,khd->qhd", torch.softmax(z, -1), vv).reshape(n, nq * d))
    ref = torch.cat(ref)
    assert bool(out[T].isnan().all())
    torch.testing.assert_close(out[:T].double().cpu(), ref, atol=4e-6 if dtype == torch.float32 else 2.0 ** -8 * float(ref.abs().max()),
                               rtol=2.0 ** -8 if dtype == torch.bfloat16 else 1e-5)


def test_attention_tokens_scores_beyond_float32():
    """A run of keys whose scores are all minus infinity leaves what the other keys give; a token with no other keys gets zeros
    (as from attention_simt)."""
    from mini_hisparse_b200.parts.attention import AttentionShape, plan_decode

    lengths, d, P_ = [40, 20, 600], 32, 32
    need = [-(-n // P_) for n in lengths]
    table = torch.full((3, max(need)), -1, dtype=torch.int32)
    for i, n in enumerate(need):
        table[i, :n] = torch.arange(sum(need[:i]), sum(need[:i]) + n)
    cache = torch.randn(sum(need), 2, 1, P_, d, generator=torch.Generator().manual_seed(1))
    q = torch.zeros(3, 2, d)
    q[..., 0], q[:, 1, 0] = 1e30, -1e30
    cache[:, 0, ..., 0] = -1e30                 # -inf for the first head, inf for the second
    cache[[1, 4], 0, :, :, 0] = 0.0             # the second page of the first and of the third request
    plan = plan_decode(AttentionShape(2, 1), np.asarray(lengths) - 1, 1)
    outs = []
    for tokens in (True, False):
        out, items = torch.empty(3, 2 * d, device=DEV), torch.from_numpy(plan.items).to(DEV).reshape(-1)
        parts = torch.zeros(1, 2, d, device=DEV), torch.zeros(1, 2, 2, device=DEV)
        tpr, pos = torch.zeros(3, dtype=torch.int32, device=DEV), torch.tensor(lengths, dtype=torch.int32, device=DEV) - 1
        if tokens:
            K().attention_tokens(q.to(DEV), cache.to(DEV), out, *parts, items, 3, table.to(DEV), tpr, nq=2, nkv=1, d=d, page_size=P_)
        else:
            K().attention_simt(q.to(DEV), cache.to(DEV), out, *parts, items, 3, 3, pos, table.to(DEV), tpr, nq=2, nkv=1, d=d, page_size=P_)
        outs.append(out.view(3, 2, d).cpu())
    got, ref = outs
    assert bool(got[:, 0].isfinite().all()) and bool((got[1, 0] == 0).all())
    torch.testing.assert_close(got[:, 0], ref[:, 0], atol=1e-5, rtol=1e-5)
    for n, page in ((8, 1), (32, 4)):           # the mean of the keys whose scores are finite (zero)
        torch.testing.assert_close(got[0 if page == 1 else 2, 0], cache[page, 1, 0, :n].mean(0), atol=1e-5, rtol=1e-5)


@pytest.mark.parametrize("nq,nkv,d,P_,nsplit", [(3, 1, 32, 32, 1), (4, 2, 16, 16, 3), (28, 4, 128, 16, 1), (16, 4, 64, 5, 4), (8, 1, 100, 7, 2),
                                                (5, 5, 4, 1, 1)])
@pytest.mark.parametrize("window", [None, 70])
@pytest.mark.parametrize("dtype", DTYPES)
def test_attention_tokens(nq, nkv, d, P_, nsplit, window, dtype):
    """Decoded tokens on the CUDA cores with the keys dealt to warps: histories around a warp's run of 32 keys, half a round and
    one and two rounds of 512 (the second fetches its rows ahead), odd pages, splits (empty ones too), a window, against 64 bits."""
    from mini_hisparse_b200.parts.attention import AttentionShape, plan_decode

    assert K().attention_tokens_supports(nq, nkv, d)
    g = torch.Generator().manual_seed(nq * d + nsplit)
    lengths = [1, 31, 32, 33, 255, 256, 257, 511, 512, 513, 600, 1025]
    B, need = len(lengths), [-(-n // P_) for n in lengths]
    order = torch.randperm(sum(need), generator=g).tolist()
    table = torch.full((B, max(need) + 1), -1, dtype=torch.int32)
    for i, n in enumerate(need):
        table[i, :n] = torch.tensor([order.pop() for _ in range(n)])
    cache, q = torch.randn(sum(need), 2, nkv, P_, d, generator=g).to(dtype), torch.randn(B, nq, d, generator=g).to(dtype)
    plan = plan_decode(AttentionShape(nq, nkv, window), np.asarray(lengths) - 1, nsplit)
    out = torch.full((B + 1, nq * d), float("nan"), dtype=dtype, device=DEV)
    part_acc, part_ml = (torch.full((max(1, plan.part_rows), nq, n), float("nan"), device=DEV) for n in (d, 2))
    tpr, tns = (torch.from_numpy(y).to(DEV) for y in (plan.tok_part_row, plan.tok_nsplit))
    K().attention_tokens(q.to(DEV), cache.to(DEV), out[:B], part_acc, part_ml, torch.from_numpy(plan.items).to(DEV).reshape(-1),
                         len(plan.items), table.to(DEV), tpr, nq=nq, nkv=nkv, d=d, page_size=P_)
    if nsplit > 1:
        K().attention_combine(part_acc, part_ml, tpr, tns, out[:B], nq=nq, d=d)
    ref = torch.empty(B, nq, d, dtype=torch.float64)
    for i, n in enumerate(lengths):
        kv = cache[table[i, :need[i]].long()].double().permute(1, 0, 3, 2, 4).reshape(2, -1, nkv, d)[:, max(0, n - (window or n)): n]
        kk, vv = (y.repeat_interleave(nq // nkv, 1) for y in kv)
        ref[i] = torch.einsum("hk,khd->hd", torch.softmax(torch.einsum("hd,khd->hk", q[i].double(), kk) * d ** -0.5, 1), vv)
    assert bool(out[B].isnan().all())
    torch.testing.assert_close(out[:B].double().cpu().view(B, nq, d), ref, atol=2e-6 if dtype == torch.float32 else 2.0 ** -8 * float(ref.abs().max()),
                               rtol=2.0 ** -8 if dtype == torch.bfloat16 else 1e-5)


@pytest.mark.parametrize("nq,nkv,d,P_,dtype", [
    (3, 1, 16, 16, torch.float32), (7, 7, 20, 5, torch.float32), (4, 2, 23, 3, torch.float32), (28, 4, 128, 16, torch.float32),
    (18, 1, 256, 1, torch.float32), (5, 5, 184, 64, torch.float32), (4, 2, 24, 16, torch.bfloat16), (4, 2, 20, 7, torch.bfloat16),
    (6, 1, 256, 16, torch.bfloat16)])
def test_attention_simt_staging(nq, nkv, d, P_, dtype):
    """The CUDA-core kernel's ways to stage a tile: 16-byte pieces or single elements (widths that are no whole number of
    pieces), two buffers or one (wide rows), with no key, one, a tile's edge and many tiles, and key splits."""
    specs = [(0, 1), (30, 1), (31, 1), (32, 2), (63, 1), (200, 17), (630, 1)]
    out, ref, plan = run_attention(nq, nkv, d, P_, specs, dtype)
    assert plan.part_rows > 1
    torch.testing.assert_close(out, ref, **tol(dtype, 4))
    out, ref, _ = run_attention(nq, nkv, d, P_, specs, dtype, window=33, fixed_nsplit=3)
    torch.testing.assert_close(out, ref, **tol(dtype, 4))


@pytest.mark.parametrize("nq,nkv,d,P_,dtype,window,digest", [
    (4, 2, 16, 16, torch.float32, None, "ff3db8955cc0fb31"), (3, 1, 32, 32, torch.float32, None, "eacb959b9b6a0da5"),
    (4, 2, 23, 3, torch.float32, None, "c8026b0b6d11cead"), (6, 2, 24, 16, torch.bfloat16, 33, "0e40358704170298"),
    (6, 1, 256, 16, torch.bfloat16, None, "6dc225df5a5a1fd7")])
def test_attention_simt_bits(nq, nkv, d, P_, dtype, window, digest):
    """The bits of the CUDA-core kernel's outputs: a digest of what the kernel gave that staged one tile at a time, element by
    element.  However tiles are staged, scores, maxima and sums are taken in that kernel's order (a tile's weights are added
    across the warp before they meet the running sum)."""
    out, _, plan = run_attention(nq, nkv, d, P_, [(0, 1), (30, 1), (31, 1), (63, 1), (200, 17), (250, 1)], dtype, window=window)
    assert plan.part_rows == 0 and hashlib.sha256(out.numpy().tobytes()).hexdigest()[:16] == digest


@pytest.mark.parametrize("nq,nkv,d,P_", [(4, 2, 32, 16), (3, 1, 32, 32), (28, 4, 128, 16), (20, 1, 96, 8),
                                          (6, 3, 64, 7), (40, 2, 128, 16)])
def test_attention_tensor_core_portions_and_decode_mixed(nq, nkv, d, P_):
    """The mma kernel: long portions (64-row tiles), short ones (16-row tiles, warps split the
    keys), portions that start inside a page, and groups larger than a tile."""
    specs = [(0, 137), (45, 19), (130, 1), (63, 2), (200, 70), (0, 1), (5, 16)]
    out, ref, plan = run_attention(nq, nkv, d, P_, specs, torch.bfloat16, kernel="mma")
    assert plan.n_small and plan.n_big
    torch.testing.assert_close(out, ref, **tol(torch.bfloat16, 2))


@pytest.mark.parametrize("nq,nkv,d,P_", [(4, 2, 64, 16), (3, 1, 128, 32), (28, 4, 128, 16), (20, 1, 64, 8),
                                          (6, 3, 128, 64), (256, 2, 128, 16), (40, 2, 128, 4)])
def test_attention_tcgen05_long_portions(nq, nkv, d, P_):
    """The tcgen05 kernel (128-row tiles, S and the O tile in tensor memory) on long portions that
    start at 0 and inside a page, beside short ones that go to the 16-row kernel."""
    specs = [(0, 300), (45, 19), (130, 1), (200, 170), (0, 1), (77, 129)]
    out, ref, plan = run_attention(nq, nkv, d, P_, specs, torch.bfloat16, kernel="tc")
    assert plan.n_small and plan.n_big
    torch.testing.assert_close(out, ref, **tol(torch.bfloat16, 2))


@pytest.mark.parametrize("nq,nkv,d,P_", [(28, 4, 128, 16), (8, 8, 64, 32), (40, 8, 128, 16)])
def test_attention_tcgen05_long_tiles_split_along_the_keys(nq, nkv, d, P_):
    """Portions of some dozens of tokens far into long prompts: fewer 128-row tiles than SMs, so the
    planner splits them along the keys and attention_combine merges the parts; beside them decode
    tokens whose splits the 16-row kernel merges itself."""
    specs = [(3000, 100), (2500, 1), (700, 1), (1800, 40)]
    out, ref, plan = run_attention(nq, nkv, d, P_, specs, torch.bfloat16, kernel="tc")
    assert plan.big_split and plan.n_small
    assert int((plan.items[plan.n_small:, 7] >= 0).sum()) > 0
    torch.testing.assert_close(out, ref, **tol(torch.bfloat16, 2))


@pytest.mark.parametrize("kernel", ["mma", "tc"])
def test_attention_tensor_core_splits_window_and_far_key(kernel):
    bf = torch.bfloat16
    for seed in (0, 1):      # merged inside the kernel, and by attention_combine
        out, ref, plan = run_attention(28, 4, 128, 16, [(700, 1), (33, 1), (1023, 1), (0, 1), (300, 2)], bf,
                                       fixed_nsplit=5, kernel=kernel, seed=seed)
        assert plan.part_rows == 30
        torch.testing.assert_close(out, ref, **tol(bf, 2))
    out, ref, plan = run_attention(40, 2, 64, 16, [(500, 1), (90, 3)], bf, fixed_nsplit=3, kernel=kernel)
    torch.testing.assert_close(out, ref, **tol(bf, 2))          # groups of 20 heads: two chunks per token
    out, ref, plan = run_attention(8, 2, 64, 16, [(2000, 1)], bf, kernel=kernel)
    assert plan.part_rows > 1
    torch.testing.assert_close(out, ref, **tol(bf, 2))
    for window in (1, 5, 16, 40, 64, 65):
        out, ref, _ = run_attention(4, 2, 64, 16, [(0, 150), (77, 3), (100, 1)], bf, window=window, kernel=kernel)
        torch.testing.assert_close(out, ref, **tol(bf, 2))

    def edit(qs, ks, vs, cache, table):
        d = qs[0].shape[-1]
        direction = torch.zeros(d)
        direction[5] = 1.0
        for h in range(qs[0].shape[1]):
            qs[0][-1, h] = direction * 60.0
        ks[0][3, :] = (direction * 8.0).to(ks[0].dtype)
        cache[int(table[0, 0]), 0, :, 3] = ks[0][3].to(cache.device)
    out, ref, _ = run_attention(4, 2, 64, 16, [(640, 1)], bf, edit=edit, kernel=kernel)
    torch.testing.assert_close(out, ref, **tol(bf, 2))
    out2, ref2, _ = run_attention(4, 2, 64, 16, [(0, 641)], bf, edit=edit, kernel=kernel)
    torch.testing.assert_close(out2, ref2, **tol(bf, 2))


@pytest.mark.parametrize("d,P_", [(64, 16), (128, 32), (128, 4)])
@pytest.mark.parametrize("hist", [0, 63, 64, 130, 191, 192, 300, 700, 1500])
def test_attention_tma_few_ctas(d, P_, hist):
    """Few CTAs with few or many tiles each: from less than one tile to several rounds of the ring of stages, unsplit and
    split, decode tokens and a short portion."""
    for nsplit in (1, 3):
        out, ref, plan = run_attention(6, 2, d, P_, [(hist, 1), (hist, 5)], torch.bfloat16, fixed_nsplit=nsplit, kernel="tc")
        assert len(plan.items) * 2 <= 148 and plan.n_small
        torch.testing.assert_close(out, ref, **tol(torch.bfloat16, 2))


@pytest.mark.parametrize("d,P_", [(64, 16), (128, 32)])
@pytest.mark.parametrize("nsplit", [1, 3])
@pytest.mark.parametrize("ext", [False, True])
def test_attention_tma_alone_and_in_a_busy_batch(d, P_, nsplit, ext):
    """A launch with more CTAs than SMs (64 decode tokens and a short portion), against the oracle, and its first segments
    launched alone: the same bits, whatever else is in the launch.  ``ext``: with a sink, a cap and a gate."""
    from mini_hisparse_b200.parts.attention import AttentionShape, plan_attention

    nq, nkv, bf = 8, 4, torch.bfloat16
    specs = [(130, 1), (64, 1)] + [(i % 150, 1) for i in range(62)] + [(70, 5)]
    cache, table, segments, qs, ks, vs, positions = paged_case(nq, nkv, d, P_, specs, bf)
    T = sum(n for _, n in specs)
    plan = plan_attention(AttentionShape(nq, nkv, None, 128), segments, T, 148, fixed_nsplit=nsplit)
    assert not plan.n_big and plan.n_small * nkv > 148
    q = torch.cat([qq[h:] for qq, (h, n) in zip(qs, specs)]).reshape(T, nq * d).to(DEV)
    sink, gate = (torch.randn(*n, generator=torch.Generator().manual_seed(d)).to(DEV) for n in ((nq,), (T, nq * d)))
    status = torch.zeros(1, dtype=torch.int32, device=DEV)

    def run(items):
        out = torch.full((T, nq * d), float("nan"), dtype=bf, device=DEV)
        rows = max(1, plan.part_rows)
        part_acc, part_ml = torch.full((rows, nq, d), float("nan"), device=DEV), torch.full((rows, nq, 2), float("nan"), device=DEV)
        counters = torch.zeros(T * nkv, dtype=torch.int32, device=DEV)
        opts = dict(sink=sink, gate=gate, softcap=20.0) if ext else {}
        (K().attention_tma_ext if ext else K().attention_tma)(
            q, cache, out, part_acc, part_ml, torch.from_numpy(items).to(DEV).reshape(-1), len(items), 16, positions, table,
            torch.from_numpy(plan.tok_part_row).to(DEV), nq=nq, nkv=nkv, d=d, page_size=P_,
            tok_nsplit=torch.from_numpy(plan.tok_nsplit).to(DEV), counters=counters, status=status, **opts)
        assert int(status) == 0 and int(counters.abs().sum()) == 0
        return out

    out = run(plan.items)
    few = plan.items[plan.items[:, 0] < 2]                      # the items of the first two segments
    assert len(few) * nkv <= 148
    assert torch.equal(run(few)[:2], out[:2])
    ref = []
    for qq, kk, vv, (h, n) in zip(qs, ks, vs, specs):
        qq, kk, vv = (y.double() for y in (qq, kk, vv))
        kk, vv = (y.repeat_interleave(nq // nkv, 1) for y in (kk, vv))
        z = torch.einsum("qhd,khd->hqk", qq[h:], kk) * d ** -0.5
        z = 20.0 * torch.tanh(z / 20.0) if ext else z
        z.masked_fill_(torch.arange(h + n) > torch.arange(h, h + n)[:, None], -math.inf)
        if ext:
            z = torch.cat((z, sink.cpu().double()[:, None, None].expand(-1, n, 1)), -1)
        ref.append(torch.einsum("hqk,khd->qhd", torch.softmax(z, -1)[..., :h + n], vv).reshape(n, nq * d))
    ref = torch.cat(ref)
    ref = ref * torch.sigmoid(gate.cpu().double()) if ext else ref
    torch.testing.assert_close(out.double().cpu(), ref, **tol(bf, 2))


@pytest.mark.parametrize("nq,nkv,d,P_,nsplit,shared,per_head", [(8, 4, 64, 16, 2, False, False), (28, 4, 128, 32, 8, False, False),
                                                                (16, 1, 128, 16, 16, True, True), (3, 1, 64, 64, 5, False, True),
                                                                (10, 1, 128, 4, 5, True, False), (16, 16, 128, 16, 7, False, False)])
@pytest.mark.parametrize("window", [None, 100])
def test_attention_tma_splits_merged_in_a_cluster(nq, nkv, d, P_, nsplit, shared, per_head, window):
    """Decoded tokens whose key splits a thread-block cluster merges: with a sink, a cap and a gate, histories with empty
    splits among them, bfloat16 and float32 outputs, the gate on and off 16 bytes.  The partial buffers and counters stay
    untouched."""
    from mini_hisparse_b200.parts.attention import AttentionShape, plan_decode

    bf = torch.bfloat16
    assert K().attention_tma_max_clusters(d, nq // nkv, nsplit) > 0
    g = torch.Generator().manual_seed(nq * d + nsplit)
    lengths = [1, 63, 64, 65, 130, 333, 700]
    B, width = len(lengths), 800 // P_ + 1
    need = [-(-n // P_) for n in lengths]
    order = torch.randperm(sum(need), generator=g).tolist()
    table = torch.full((B, width), -1, dtype=torch.int32)
    for i, n in enumerate(need):
        table[i, :n] = torch.tensor([order.pop() for _ in range(n)])
    planes = 1 if shared else 2
    cache = torch.randn(sum(need), planes, nkv, P_, d, generator=g).to(bf)
    q = torch.randn(B, nq, d, generator=g).to(bf)
    sink, gate = torch.randn(nq, generator=g), torch.randn(2, B, 2 + (nq if per_head else nq * d), generator=g)
    plan = plan_decode(AttentionShape(nq, nkv, window, 128), np.asarray(lengths) - 1, nsplit)
    z = gate.double().sum(0)
    for first in (0, 1):            # the gate's first column
        cols = z[:, first: first + (nq if per_head else nq * d)].view(B, nq, -1)
        ref = torch.empty(B, nq, d, dtype=torch.float64)
        for i, n in enumerate(lengths):
            kv = cache[table[i, :need[i]].long()].double().permute(1, 0, 3, 2, 4).reshape(planes, -1, nkv, d)[:, max(0, n - (window or n)): n]
            kk, vv = (kv[j].repeat_interleave(nq // nkv, 1) for j in (0, planes - 1))
            x = 20.0 * torch.tanh(torch.einsum("hd,khd->hk", q[i].double(), kk) * d ** -0.5 / 20.0)
            w = torch.softmax(torch.cat((x, sink.double()[:, None]), 1), 1)[:, :-1]
            ref[i] = torch.einsum("hk,khd->hd", w, vv) * torch.sigmoid(cols[i])
        for dtype in (bf, torch.float32):
            out = torch.full((B + 1, nq * d), float("nan"), dtype=dtype, device=DEV)
            part, counters = torch.full((B * nsplit, nq, d), 7.0, device=DEV), torch.zeros(B * nkv, dtype=torch.int32, device=DEV)
            status = torch.zeros(1, dtype=torch.int32, device=DEV)
            gd = gate.to(DEV)
            K().attention_tma_ext(
                q.to(DEV), cache.to(DEV), out[:B], part, part[..., :2].contiguous(), torch.from_numpy(plan.items).to(DEV).reshape(-1),
                len(plan.items), 16, torch.tensor(lengths, dtype=torch.int32, device=DEV) - 1, table.to(DEV),
                torch.from_numpy(plan.tok_part_row).to(DEV), nq=nq, nkv=nkv, d=d, page_size=P_, window=window or 0, sink=sink.to(DEV),
                gate=gd[0][:, first:], gate_nsplit=2, gate_split_stride=gd.stride(0), gate_per_head=per_head, shared_kv=shared,
                softcap=20.0, tok_nsplit=torch.from_numpy(plan.tok_nsplit).to(DEV), counters=counters, status=status, cluster=nsplit)
            assert int(status) == 0 and int(counters.abs().sum()) == 0 and bool((part == 7.0).all()) and bool(out[B].isnan().all())
            got = out[:B].double().cpu().view(B, nq, d)
            # weights in 16 bits, float32 sums; a bfloat16 output adds its own rounding
            torch.testing.assert_close(got, ref, atol=1e-4 if dtype == torch.float32 else 2.0 ** -8 * float(ref.abs().max()), rtol=2.0 ** -8 if dtype == bf else 0)


@pytest.mark.parametrize("kind,dtype", [("plain", torch.bfloat16), ("ext", torch.bfloat16), ("ext", torch.float32)])
@pytest.mark.parametrize("nsplit,merge", [(1, "none"), (3, "counters"), (3, "later"), (2, "cluster")])
def test_attention_tma_buffers_off_their_vectors(kind, dtype, nsplit, merge):
    """Outputs and partial buffers that start an element off 8 and 16 bytes get what aligned ones get, bit for bit."""
    from mini_hisparse_b200.parts.attention import AttentionShape, plan_decode

    if (kind, merge) == ("plain", "cluster"):
        pytest.skip("the kernel without options merges in no cluster")
    nq, nkv, d, P_, lengths = 6, 2, 64, 16, [1, 70, 260]
    g, B = torch.Generator().manual_seed(nsplit), len(lengths)
    table = torch.arange(B * 17, dtype=torch.int32, device=DEV).view(B, 17)
    cache = torch.randn(B * 17, 2, nkv, P_, d, generator=g).bfloat16().to(DEV)
    q = torch.randn(B, nq * d, generator=g).bfloat16().to(DEV)
    plan = plan_decode(AttentionShape(nq, nkv, None, 128), np.asarray(lengths) - 1, nsplit)
    items, pos = torch.from_numpy(plan.items).to(DEV).reshape(-1), torch.tensor(lengths, dtype=torch.int32, device=DEV) - 1
    tpr, tns = (torch.from_numpy(y).to(DEV) for y in (plan.tok_part_row, plan.tok_nsplit))
    rows, results = max(1, plan.part_rows), []
    for off in (0, 1):
        out = torch.full((B * nq * d + 8,), float("nan"), dtype=dtype, device=DEV)
        acc, ml = torch.full((rows * nq * d + 8,), 3.0, device=DEV), torch.full((rows * nq * 2 + 8,), 3.0, device=DEV)
        o = out[off: off + B * nq * d].view(B, nq * d)
        pa, pm = acc[off: off + rows * nq * d].view(rows, nq, d), ml[off: off + rows * nq * 2].view(rows, nq, 2)
        counters, status = torch.zeros(B * nkv, dtype=torch.int32, device=DEV), torch.zeros(1, dtype=torch.int32, device=DEV)
        extra = dict(cluster=nsplit) if merge == "cluster" else dict(counters=counters) if merge == "counters" else {}
        call = K().attention_tma_ext if kind == "ext" else K().attention_tma
        call(q, cache, o, pa, pm, items, len(plan.items), 16, pos, table, tpr, nq=nq, nkv=nkv, d=d, page_size=P_, tok_nsplit=tns,
             status=status, **extra)
        assert int(status) == 0 and bool(out[off + B * nq * d:].isnan().all()) and bool((acc[off + rows * nq * d:] == 3.0).all())
        results.append([pa.cpu(), pm.cpu()] if merge == "later" else [o.cpu()])
    for x, y in zip(*results):      # an empty split's partials have a maximum of minus infinity
        assert torch.equal(x, y) and not bool(x.isnan().any())


@pytest.mark.parametrize("ext", [False, True])
@pytest.mark.parametrize("n", [1, 2, 16])
def test_attention_tma_early_keys_behind_the_append(ext, n):
    """``fresh``: keys older than the step are read before the kernel that appends the step's own is done.  Straight behind
    that kernel, with histories around the edges of tiles and of what counts as fresh, the result is that of a launch that
    waits for every key."""
    from mini_hisparse_b200.parts.attention import AttentionShape, plan_attention

    nq, nkv, d, P_, bf = 8, 2, 64, 16, torch.bfloat16
    specs = [(h, n) for h in (0, 15, 16, 63, 64, 79, 80, 200)]
    cache, table, segments, _, _, _, positions = paged_case(nq, nkv, d, P_, specs, bf)
    T = n * len(specs)
    plan = plan_attention(AttentionShape(nq, nkv, None, 128), segments, T, 148, fixed_nsplit=1)
    assert plan.n_small == len(plan.items)
    items, status = torch.from_numpy(plan.items).to(DEV).reshape(-1), torch.zeros(1, dtype=torch.int32, device=DEV)
    seg = torch.arange(len(specs), dtype=torch.int32, device=DEV).repeat_interleave(n)
    qkv = rnd(T, (nq + 2 * nkv) * d, seed=3)
    parts = torch.zeros(1, nq, d, device=DEV), torch.zeros(1, nq, 2, device=DEV)
    tpr, tns = (torch.from_numpy(y).to(DEV) for y in (plan.tok_part_row, plan.tok_nsplit))
    launch = K().attention_tma_ext if ext else K().attention_tma
    results = []
    for fresh in (0, 16) * 10:
        pool, q, out = cache.clone(), torch.empty(T, nq * d, dtype=bf, device=DEV), torch.empty(T, nq * d, dtype=bf, device=DEV)
        K().rope_append(qkv, None, positions, seg, table, None, q, pool, nq=nq, nkv=nkv, d=d, page_size=P_, status=status)
        launch(q, pool, out, *parts, items, plan.n_small, 16, positions, table, tpr, nq=nq, nkv=nkv, d=d, page_size=P_, tok_nsplit=tns,
               status=status, fresh=fresh)
        results.append(out)
    assert int(status) == 0 and all(torch.equal(y, results[0]) for y in results)


@pytest.mark.parametrize("nq,nkv,d,P_,nsplit,qkv_nsplit,rdim,interleaved,window,ngroups", [
    (28, 4, 128, 16, 8, 8, 128, False, None, 1),       # the benchmark's shape: 7 heads per KV head, clusters of 8
    (28, 4, 128, 16, 16, 3, 128, False, None, 1),      # clusters of 16
    (3, 1, 64, 32, 1, 1, 64, False, None, 1),          # one share: nothing to merge
    (32, 2, 128, 8, 4, 2, 64, True, None, 1),          # 16 heads per KV head, interleaved pairs on half the head
    (8, 8, 64, 64, 3, 4, 0, False, None, 1),           # no rotation, one head per KV head, pages of a whole tile
    (12, 4, 128, 4, 6, 1, 96, False, 300, 1),          # a window, tiny pages; 3 heads over 6 shares: some CTAs own no row
    (20, 4, 64, 16, 3, 5, 64, False, None, 1),         # 5 heads over 3 shares: a CTA owns two rows
    (28, 4, 128, 16, 4, 2, 128, False, None, 3),       # three clusters of 4 per token and KV head, merged by attention_combine
    (12, 4, 128, 4, 2, 1, 96, False, 300, 5),          # five clusters of 2, a window: most groups of short histories are empty
    (20, 4, 64, 16, 3, 5, 64, True, None, 2),          # two clusters of 3, a CTA owns two rows
    (3, 1, 64, 32, 1, 1, 64, False, None, 4),          # four clusters of one CTA
])
def test_attention_decode_fused(nq, nkv, d, P_, nsplit, qkv_nsplit, rdim, interleaved, window, ngroups):
    """The decode kernel that does everything between the q/k/v product and the output projection:
    sums the product's parts, adds the bias, rotates, appends k and v to their pages, attends over
    the cache and merges the key shares in its cluster (with several clusters per token and KV head,
    every cluster leaves a part and attention_combine merges them).  Histories of 0, a few, one tile,
    and many keys, some ending at a page's or a tile's edge; one far key among hundreds stands out."""
    check_attention_decode([0, 5, 63, 64, 127, 700, 1023, 333], nq, nkv, d, P_, nsplit, qkv_nsplit, rdim, interleaved,
                           window, ngroups)


def test_attention_decode_fused_more_clusters_than_fit():
    """A batch of 90 tokens with uneven histories and three shares each: 1,080 CTAs in 360 clusters, several
    rounds of them (what the planner chooses for a large batch that would else wait for its longest
    history)."""
    g = torch.Generator().manual_seed(11)
    histories = torch.randint(0, 900, (90,), generator=g).tolist()
    histories[7], histories[50] = 2300, 1999
    check_attention_decode(histories, 28, 4, 128, 16, 3, 2, 128, False, None, 1)


def check_attention_decode(histories, nq, nkv, d, P_, nsplit, qkv_nsplit, rdim, interleaved, window, ngroups):
    bf = torch.bfloat16
    T = len(histories)
    theta = 10000.0
    g = torch.Generator().manual_seed(3)
    width_all = (nq + 2 * nkv) * d
    parts = (torch.randn(qkv_nsplit, T, width_all, generator=g) / math.sqrt(qkv_nsplit)).to(DEV)
    bias = (torch.randn(width_all, generator=g) * 0.1).to(DEV)
    positions = torch.tensor(histories, dtype=torch.int32, device=DEV)
    full = (parts.sum(0) + bias).cpu()
    q = plain_rotation(full[:, : nq * d].view(T, nq, d), positions.cpu(), theta, rdim, interleaved).to(bf).float()
    pages_of = [-(-(h + 1) // P_) for h in histories]
    pool = sum(pages_of) + 5
    perm = torch.randperm(pool, generator=g).tolist()
    cache = torch.randn(pool, 2, nkv, P_, d, generator=g).to(bf).to(DEV)          # stale junk everywhere
    table = torch.full((T, max(pages_of)), -1, dtype=torch.int32)
    ks, vs = [], []
    for i, h in enumerate(histories):
        pages = [perm.pop() for _ in range(pages_of[i])]
        table[i, : len(pages)] = torch.tensor(pages)
        k = torch.randn(h, nkv, d, generator=g).to(bf)
        v = torch.randn(h, nkv, d, generator=g).to(bf)
        if h > 600:          # one far key that the first head of every group looks for: its score stands out
            k[37] = (0.5 * q[i, :: nq // nkv]).to(bf)
        for t in range(h):
            cache[pages[t // P_], 0, :, t % P_] = k[t].to(DEV)
            cache[pages[t // P_], 1, :, t % P_] = v[t].to(DEV)
        ks.append(k), vs.append(v)
    table = table.to(DEV)
    inv = (theta ** (-torch.arange(0, rdim, 2).float() / rdim)).to(DEV) if rdim else None
    before = cache.clone()
    out = torch.full((T, nq * d), float("nan"), dtype=bf, device=DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    assert K().attention_decode_supports(d, P_, nq // nkv, nsplit, rdim)
    extra = {}
    if ngroups > 1:
        extra = dict(ngroups=ngroups, part_acc=torch.full((T * ngroups, nq, d), float("nan"), device=DEV),
                     part_ml=torch.full((T * ngroups, nq, 2), float("nan"), device=DEV))
    K().attention_decode(parts, bias, inv, cache, out, positions, table, nq=nq, nkv=nkv, d=d, page_size=P_,
                         nsplit=nsplit, qkv_nsplit=qkv_nsplit, qkv_split_stride=parts.stride(0), rotary_dim=rdim,
                         interleaved=interleaved, window=window or 0, status=status, **extra)
    assert int(status) == 0
    k_new = plain_rotation(full[:, nq * d: (nq + nkv) * d].view(T, nkv, d), positions.cpu(), theta, rdim, interleaved).to(bf)
    v_new = full[:, (nq + nkv) * d:].view(T, nkv, d).to(bf)
    touched = torch.zeros(pool, P_, dtype=torch.bool)
    for i, h in enumerate(histories):
        k_all = torch.cat((ks[i], k_new[i: i + 1])).float()
        v_all = torch.cat((vs[i], v_new[i: i + 1])).float()
        q_all = torch.zeros(h + 1, nq, d)
        q_all[h] = q[i]
        ref = P.causal_attention(q_all, k_all, v_all, window=window)[h].reshape(-1)
        torch.testing.assert_close(out[i].float().cpu(), ref, **tol(bf, 2))
        page = int(table[i, h // P_])
        torch.testing.assert_close(cache[page, 0, :, h % P_].float().cpu(), k_new[i].float(), **tol(bf, 4))
        torch.testing.assert_close(cache[page, 1, :, h % P_].float().cpu(), v_new[i].float(), **tol(bf, 4))
        touched[page, h % P_] = True
    # nothing but the tokens' own slots was written
    same = (cache == before).all(-1).all(1).all(1).cpu()        # [pool, P]
    assert bool(same[~touched].all())


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("nq,nkv,d,P_", [(4, 2, 16, 16), (3, 1, 32, 32), (10, 2, 48, 16), (28, 4, 128, 16),
                                          (20, 1, 80, 8), (2, 2, 256, 16), (6, 3, 112, 7)])
def test_attention_prefill_portions_and_decode_mixed(dtype, nq, nkv, d, P_):
    # a whole prompt, a portion at an offset inside a page, a single token, a 2-token portion
    specs = [(0, 37), (45, 19), (130, 1), (63, 2)]
    out, ref, plan = run_attention(nq, nkv, d, P_, specs, dtype)
    torch.testing.assert_close(out, ref, **tol(dtype, 2))


@pytest.mark.parametrize("dtype", DTYPES)
def test_attention_split_keys_and_combine(dtype):
    specs = [(700, 1), (33, 1), (1023, 1), (0, 1)]
    out, ref, plan = run_attention(28, 4, 128, 16, specs, dtype, fixed_nsplit=5)
    assert plan.part_rows == 20 and (plan.items[:, 7] >= 0).all()
    torch.testing.assert_close(out, ref, **tol(dtype, 2))
    out, ref, plan = run_attention(8, 2, 64, 16, [(2000, 1)], dtype)      # the planner splits by itself
    assert plan.part_rows > 1
    torch.testing.assert_close(out, ref, **tol(dtype, 2))


@pytest.mark.parametrize("dtype", DTYPES)
def test_attention_finds_one_far_key_among_hundreds(dtype):
    """Random keys give near-uniform weights, which would hide a missed page.  Here the query of
    the last token matches key 3 (first page) with a large score: the output must be V[3]."""
    def edit(qs, ks, vs, cache, table):
        d = qs[0].shape[-1]
        direction = torch.zeros(d)
        direction[5] = 1.0
        for h in range(qs[0].shape[1]):
            qs[0][-1, h] = direction * 60.0
        ks[0][3, :] = (direction * 8.0).to(ks[0].dtype)
        page = int(table[0, 0])
        cache[page, 0, :, 3] = ks[0][3].to(cache.device)
    out, ref, _ = run_attention(4, 2, 64, 16, [(640, 1)], dtype, edit=edit)
    torch.testing.assert_close(out, ref, **tol(dtype, 2))
    # and the reference itself is V[3] there, up to the tail of the softmax
    out2, ref2, _ = run_attention(4, 2, 64, 16, [(0, 641)], dtype, edit=edit)
    torch.testing.assert_close(out2[-1], ref2[-1], **tol(dtype, 2))
    torch.testing.assert_close(out[-1], out2[-1], **tol(dtype, 2))


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("window", [1, 5, 16, 40])
def test_attention_window_edge(dtype, window):
    """Keys exactly at the window's edge: position - window + 1 is the first key kept."""
    specs = [(0, 50), (77, 3), (100, 1)]
    out, ref, _ = run_attention(4, 2, 32, 16, specs, dtype, window=window)
    torch.testing.assert_close(out, ref, **tol(dtype, 2))


def test_attention_refuses_what_it_cannot_do():
    from mini_hisparse_b200.kernels.api import KernelError
    from mini_hisparse_b200.parts.attention import GQAttention
    from mini_hisparse_b200.parts.spec import PartSpec

    pos = PartSpec.make("rotary", head_dim=40, theta=1e4)
    with pytest.raises(ValueError, match="head_dim 40"):
        GQAttention(PartSpec.make("gq_attention", hidden_size=80, q_heads=2, kv_heads=2, head_dim=40, position=pos))
    with pytest.raises(KernelError, match="CPU"):
        K().embed(torch.zeros(4, 4), torch.zeros(1, dtype=torch.int32), torch.zeros(1, 4))


# ---- sampling -------------------------------------------------------------------------------------
def test_sample_greedy_lowest_index_wins():
    V = 152064 // 8 + 3
    logits = rnd(5, V, seed=3)
    logits[1, 100] = logits[1, 17000] = 50.0
    logits[2, V - 1] = 60.0
    logits[3, 0] = 60.0
    out = torch.empty(5, dtype=torch.int32, device=DEV)
    K().sample(logits, None, None, None, out)
    assert out.tolist() == logits.argmax(-1).tolist()
    assert out[1] == 100 and out[2] == V - 1 and out[3] == 0


def test_sample_temperature_equals_the_plain_draw():
    V, R = 1000, 64
    logits = rnd(R, V, seed=4, scale=2.0)
    temps = torch.tensor([0.8] * (R - 2) + [0.0, 1.5], device=DEV)
    seeds = torch.arange(R, dtype=torch.int64, device=DEV) + 11
    counters = torch.arange(R, dtype=torch.int64, device=DEV) * 3
    out = torch.empty(R, dtype=torch.int32, device=DEV)
    K().sample(logits, temps, seeds, counters, out)
    cpu = logits.cpu()
    for r in range(R):
        if float(temps[r]) == 0:
            assert int(out[r]) == int(cpu[r].argmax())
            continue
        token, margin = P.sample_temperature(cpu[r], float(temps[r]), int(seeds[r]), int(counters[r]))
        assert int(out[r]) == token or margin < 1e-5, (r, int(out[r]), token, margin)
    # the same request draws the same token whatever else is in the batch
    again = torch.empty(3, dtype=torch.int32, device=DEV)
    sel = [5, 40, 9]
    K().sample(logits[sel].contiguous(), temps[sel].contiguous(), seeds[sel].contiguous(),
               counters[sel].contiguous(), again)
    assert again.tolist() == [int(out[i]) for i in sel]


def captured_edges(graph):
    """{node: [(node in front, whether the launch allows an early start)]} of a captured graph that kept its nodes."""
    import ctypes

    cudart, n = ctypes.CDLL("libcudart.so.12"), ctypes.c_size_t(0)
    raw = ctypes.c_void_p(graph.raw_cuda_graph())
    assert cudart.cudaGraphGetEdges_v2(raw, None, None, None, ctypes.byref(n)) == 0
    front, behind, data = (ctypes.c_void_p * n.value)(), (ctypes.c_void_p * n.value)(), (ctypes.c_uint8 * (8 * n.value))()
    assert cudart.cudaGraphGetEdges_v2(raw, front, behind, data, ctypes.byref(n)) == 0
    edges = {}
    for i in range(n.value):
        edges.setdefault(behind[i], []).append((front[i], data[8 * i + 2] == 1))
    return edges


@pytest.mark.parametrize("nested", [False, True])
def test_kernels_behind_forks_and_joins_have_one_node_in_front(nested):
    """Three layers of two branches (in each a fork inside the fork, too), captured: no kernel may start beside one of two nodes
    in front, every branch is joined, and the replay gives what the launches one by one give."""
    from types import SimpleNamespace

    from mini_hisparse_b200.parts.base import fork_branch, join_branch

    branch, events = torch.cuda.Stream(), [torch.cuda.Event() for _ in range(2)]
    first = (torch.arange(8 * 256) % 7).float().view(8, 256)
    x, want = torch.empty(6, 8, 256, device=DEV), torch.zeros(6, 8, 256)
    want[1] = first

    def layers(add, fork, join):
        for _ in range(3):
            add(0, 1)
            with fork():
                add(2, 0)
                add(2, 0)
            if nested:
                add(3, 0)
                with fork():
                    add(4, 3)
                add(5, 0)
                join()
                add(3, 4)
                add(3, 5)
            add(3, 0)
            join()
            add(1, 2)
            add(1, 3)

    def on_the_gpu():
        ctx = SimpleNamespace(open_branches=[])

        @contextlib.contextmanager
        def fork():
            fork_branch(ctx, branch, events[0])
            with torch.cuda.stream(branch):
                yield
                events[1].record(branch)

        layers(lambda into, what: K().residual_add(x[into], x[what]), fork, lambda: join_branch(ctx, branch, events[1]))
        assert not ctx.open_branches

    def check(run):
        x.zero_()
        x[1].copy_(first)
        run()
        torch.cuda.synchronize()
        assert torch.equal(x.cpu(), want)

    layers(lambda into, what: want[into].add_(want[what]), contextlib.nullcontext, lambda: None)
    check(on_the_gpu)
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        on_the_gpu()
    edges = captured_edges(graph)
    assert any(early for front in edges.values() for _, early in front) and any(len(front) == 2 for front in edges.values())
    assert all(len(front) == 1 for front in edges.values() if any(early for _, early in front))
    check(graph.replay)
