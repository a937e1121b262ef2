"""Each kernel alone against a plain float64 PyTorch reference of the same
operation, at sizes other than the engine's, in float32 and bfloat16."""
import math
import random

import numpy as np
import pytest
import torch

import plain_qwen3 as P
from gpu_util import pack_meta as pack_step, split_length
from kipp_b200.engine.batch import StepEntry

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
DTYPES = [torch.float32, torch.bfloat16]


def ops():
    from kipp_b200 import kernels
    return kernels


def status():
    return torch.zeros(4, dtype=torch.int32, device=DEV)


def tol(dtype):
    return dict(rtol=2e-5, atol=2e-5) if dtype == torch.float32 else dict(rtol=2e-2, atol=2e-2)


# ------------------------------------------------------------------ embedding, norm
@pytest.mark.parametrize("dtype", DTYPES)
def test_embed_gather(dtype):
    g = torch.Generator().manual_seed(0)
    table = torch.randn(301, 72, generator=g).to(dtype).to(DEV)
    ids = torch.tensor([0, 300, 17, 17, 5], dtype=torch.int32, device=DEV)
    out = torch.empty(5, 72, dtype=torch.float32, device=DEV)
    st = status()
    ops().embed_gather(out, table, ids, st)
    assert torch.equal(out.cpu(), table.float().cpu()[ids.cpu().long()])
    assert st.tolist() == [0, 0, 0, 0]


@pytest.mark.parametrize("out_dtype", DTYPES)
@pytest.mark.parametrize("size", [40, 100, 256, 1028, 2560, 4096, 5000])
def test_rmsnorm(size, out_dtype):
    g = torch.Generator().manual_seed(size)
    x = (torch.randn(7, size, generator=g) * 3).to(DEV)
    for w_dtype in DTYPES:
        w = (1 + 0.2 * torch.randn(size, generator=g)).to(w_dtype).to(DEV)
        out = torch.empty(7, size, dtype=out_dtype, device=DEV)
        ops().rmsnorm(out, x, w, 1e-5)
        ref = P.plain_rmsnorm(x.cpu(), w.float().cpu(), 1e-5)
        assert torch.allclose(out.double().cpu(), ref, **tol(out_dtype))
    rows = torch.tensor([6, 0, 3], dtype=torch.int32, device=DEV)
    out = torch.empty(3, size, dtype=out_dtype, device=DEV)
    ops().rmsnorm(out, x, w, 1e-5, rows)
    assert torch.allclose(out.double().cpu(), ref[[6, 0, 3]], **tol(out_dtype))


@pytest.mark.parametrize("size", [24, 200, 320, 1000, 2560, 5120])
def test_rmsnorm_deferred(size):
    """x * weight alone and the sums of squares beside it; the two give the norm."""
    g = torch.Generator().manual_seed(size + 1)
    x = (torch.randn(9, size, generator=g) * 3).to(DEV)
    for w_dtype in DTYPES:
        w = (1 + 0.2 * torch.randn(size, generator=g)).to(w_dtype).to(DEV)
        for out_dtype in DTYPES:
            out = torch.empty(9, size, dtype=out_dtype, device=DEV)
            ssq = torch.full((9,), -1.0, device=DEV)
            ops().rmsnorm_deferred(out, ssq, x, w)
            assert torch.equal(out.cpu(), (x.cpu() * w.float().cpu()).to(out_dtype))       # one rounding
            assert torch.allclose(ssq.double().cpu(), (x.double().cpu() ** 2).sum(-1), rtol=1e-6)
            both = out.double().cpu() / torch.sqrt(ssq.double().cpu()[:, None] / size + 1e-5)
            assert torch.allclose(both, P.plain_rmsnorm(x.cpu(), w.float().cpu(), 1e-5), **tol(out_dtype))
    rows = torch.tensor([6, 0, 3], dtype=torch.int32, device=DEV)
    out = torch.empty(3, size, dtype=torch.bfloat16, device=DEV)
    ssq = torch.zeros(3, device=DEV)
    ops().rmsnorm_deferred(out, ssq, x, w, rows)
    assert torch.equal(out.cpu(), (x.cpu()[[6, 0, 3]] * w.float().cpu()).to(torch.bfloat16))


@pytest.mark.parametrize("rows", [591, 592, 593, 1183, 1184, 1185, 1300])
@pytest.mark.parametrize("size", [256, 1024, 1028, 2052, 4096])
def test_rmsnorm_of_many_rows(size, rows):
    """From 593 rows on (1,185 of up to 1,024 values) a block has several: each row's result has the bits it has alone."""
    g = torch.Generator().manual_seed(size + rows)
    x, w = torch.randn(rows, size, generator=g).to(DEV), torch.randn(size, generator=g).to(DEV)
    out, ssq, normed = torch.empty(rows, size, dtype=torch.bfloat16, device=DEV), torch.empty(rows, device=DEV), torch.empty(rows, size, device=DEV)
    ops().rmsnorm_deferred(out, ssq, x, w)
    ops().rmsnorm(normed, x, w, 1e-5)
    assert torch.equal(out, (x * w).bfloat16())
    for r in (0, 1, rows // 2, rows - 2, rows - 1):
        one, s, n = torch.empty(1, size, dtype=torch.bfloat16, device=DEV), torch.empty(1, device=DEV), torch.empty(1, size, device=DEV)
        ops().rmsnorm_deferred(one, s, x[r:r + 1], w)
        ops().rmsnorm(n, x[r:r + 1], w, 1e-5)
        assert torch.equal(s, ssq[r:r + 1]) and torch.equal(n, normed[r:r + 1])
    assert torch.allclose(ssq.double(), (x.double() ** 2).sum(-1), rtol=size * 2.0 ** -24)
    assert torch.allclose(normed.double().cpu(), P.plain_rmsnorm(x.cpu(), w.cpu(), 1e-5), **tol(torch.float32))


# ------------------------------------------------------------------ matrix products
def gemm_ref(a, w, epilogue, base):
    p = a.double().cpu() @ w.double().cpu().t()
    if epilogue == "swiglu":
        return P.plain_silu(p[:, 0::2]) * p[:, 1::2]
    return base.double().cpu() + p if epilogue == "add" else p


@pytest.mark.parametrize("epilogue", ["store", "add", "swiglu"])
@pytest.mark.parametrize("shape", [(1, 10, 24), (37, 130, 72), (64, 64, 16), (5, 1000, 136), (130, 66, 200)])
@pytest.mark.parametrize("dtype", DTYPES)
def test_gemm_simt(dtype, shape, epilogue):
    M, N, K = shape
    g = torch.Generator().manual_seed(M + N)
    a = torch.randn(M, K, generator=g).to(dtype).to(DEV)
    w = (torch.randn(N, K, generator=g) * 0.2).to(dtype).to(DEV)
    odt = torch.float32 if epilogue == "add" else dtype
    out = torch.randn(M, N // 2 if epilogue == "swiglu" else N, generator=g).to(odt).to(DEV)
    ref = gemm_ref(a, w, epilogue, out)
    ops().gemm(out, a, w, epilogue, impl="simt")
    assert torch.allclose(out.double().cpu(), ref, **tol(odt))


@pytest.mark.parametrize("epilogue", ["store", "add", "swiglu"])
@pytest.mark.parametrize("shape", [(130, 20), (18, 136), (66, 260), (2, 1028), (34, 2064), (9470, 36), (9474, 260)])
def test_gemm_32_bit_kernels_agree(shape, epilogue):
    """The 32-bit product's three kernels add in one order: the rows of a batch have the same bits whether 1, 3,
    16, 17, 32 (the kernel for few tokens, at its block sizes and the last count it takes), 33 or 70 of them (tiles)
    are multiplied at once, and where rows do not start on 16 bytes; from 9,472 features on a thread of the kernel for
    few tokens has two of them where there are 5 to 8 tokens, and tiles take over at 17.  The K reach from one run of 16 to
    runs that end inside a tile; the error against float64 stays under that of one chain of K roundings, K eps |a| |w|."""
    N, K = shape
    M = 70
    g = torch.Generator().manual_seed(N + K)
    a, w = torch.randn(M, K, generator=g).to(DEV), torch.randn(N, K, generator=g).to(DEV)
    base = torch.randn(M, N // 2 if epilogue == "swiglu" else N, generator=g).to(DEV)
    whole = base.clone()
    ops().gemm(whole, a, w, epilogue, impl="simt")
    if epilogue != "swiglu":
        bound = K * 2.0 ** -24 * (a.double().abs() @ w.double().abs().t()) + 2.0 ** -23 * whole.double().abs()
        assert ((whole.double().cpu() - gemm_ref(a, w, epilogue, base)).abs() <= bound.cpu()).all()
    for m in (1, 2, 3, 5, 7, 8, 9, 16, 17, 32, 33):
        some = base[:m].clone()
        ops().gemm(some, a[:m], w, epilogue, impl="simt")
        assert torch.equal(some, whole[:m]), m
    odd = torch.zeros(M, K + 1, device=DEV)[:, :K]
    odd.copy_(a)
    some = base.clone()
    ops().gemm(some, odd, w, epilogue, impl="simt")
    assert torch.equal(some, whole)


@pytest.mark.parametrize("epilogue", ["store", "add", "swiglu"])
@pytest.mark.parametrize("M,N,K", [(70, 12418, 2048), (200, 6206, 1028), (400, 3140, 520)])
def test_gemm_32_bit_tiles_of_256_features(M, N, K, epilogue):
    """Tiles of 256 features, the last of which ends in its upper half or its lower one, and of 128 for the first rows (or the kernel
    for few tokens): the same bits, within K eps |a| |w| of float64."""
    from kipp_b200.csrc.build import load_library
    features = load_library("gemm_simt").kipp_gemm_simt_tile_features
    assert features(M, N, K) == 256 and features(16, N, K) == 0 and features(64, N, K) == 128
    g = torch.Generator().manual_seed(M)
    a, w = torch.randn(M, K, generator=g).to(DEV), torch.randn(N, K, generator=g).to(DEV)
    base = torch.randn(M, N // 2 if epilogue == "swiglu" else N, generator=g).to(DEV)
    whole = base.clone()
    ops().gemm(whole, a, w, epilogue, impl="simt")
    if epilogue != "swiglu":
        bound = K * 2.0 ** -24 * (a.double().abs() @ w.double().abs().t()) + 2.0 ** -23 * whole.double().abs()
        assert ((whole.double() - (a.double() @ w.double().t() + (base.double() if epilogue == "add" else 0))).abs() <= bound).all()
    for m in (8, 16, 64):
        some = base[:m].clone()
        ops().gemm(some, a[:m], w, epilogue, impl="simt")
        assert torch.equal(some, whole[:m]), m


@pytest.mark.parametrize("dtype,shape,w_rows", [(torch.bfloat16, (5, 70, 100), 100), (torch.bfloat16, (65, 130, 37), 40),
                                                (torch.float32, (3, 66, 37), 37), (torch.float32, (70, 20, 60), 61)])
def test_gemm_simt_chain(dtype, shape, w_rows):
    """What only the general kernel takes (bfloat16, and 32-bit weights whose rows do not start on 16 bytes) is one chain
    of FMAs in the order of k.  The products of 8-bit mantissas are exact in 32 bits, so a loop of rounded additions
    gives every bit."""
    M, N, K = shape
    g = torch.Generator().manual_seed(K)
    a, w = torch.randn(M, K, generator=g).bfloat16().float(), torch.randn(N, K, generator=g).bfloat16().float()
    want = torch.zeros(M, N)
    for k in range(K):
        want = want + a[:, k:k + 1] * w[:, k]
    held = torch.zeros(N, w_rows, dtype=dtype, device=DEV)
    held[:, :K] = w
    out = torch.zeros(M, N, device=DEV)
    ops().gemm(out, a.to(dtype).to(DEV), held[:, :K], "store", impl="simt")
    assert torch.equal(out.cpu(), want)


@pytest.mark.parametrize("epilogue", ["store", "add", "swiglu"])
@pytest.mark.parametrize("splits", [2, 3, 5, 6, 7, 8])
def test_gemm_sends_partial_sums(splits, epilogue):
    """Up to 16 tokens the CTAs of a split product send their sums to the one that finishes a token: every share of tokens
    (some CTAs have none, the last ones fewer), features that end inside a tile; whole numbers come out exactly."""
    from kipp_b200.kernels import gemm_bf16
    N, K = 200, 64 * splits * 3
    g = torch.Generator().manual_seed(splits)
    a = torch.randint(-3, 4, (16, K), generator=g).to(torch.bfloat16).to(DEV)
    w = torch.randint(-2, 3, (N, K), generator=g).to(torch.bfloat16).to(DEV)
    for M in (1, 2, 3, 7, 8, 9, 15, 16):
        out = torch.randint(-5, 6, (M, N // 2 if epilogue == "swiglu" else N), generator=g).float().to(DEV)
        ref = gemm_ref(a[:M], w, epilogue, out)
        gemm_bf16.run("tc", out, a[:M], w, epilogue, M, splits=splits)
        if epilogue == "swiglu":
            assert torch.allclose(out.double().cpu(), ref, rtol=1e-5, atol=1e-4), M       # (the silu's division and exponential)
        else:
            assert torch.equal(out.double().cpu(), ref), M


@pytest.mark.parametrize("epilogue", ["store", "add", "swiglu"])
@pytest.mark.parametrize("shape", [(1, 128, 64), (8, 256, 128), (17, 250, 192), (64, 1000, 136),
                                   (100, 384, 2568), (300, 640, 520), (5, 2560, 1216), (40, 14400, 136),
                                   (100, 14400, 72)])
def test_gemm_tensor_core(shape, epilogue):
    """tcgen05 kernel: integer data must come out exactly (any wrong tile,
    swizzle or split shows), random data within bfloat16 rounding; K splits of
    1, a forced 3 and the cluster maximum 8.  The last two shapes have so many
    features that, left to itself (splits 0), a store or SwiGLU product of 33 to
    511 tokens takes the kernel with the tokens as rows."""
    from kipp_b200.kernels import gemm_bf16
    M, N, K = shape
    g = torch.Generator().manual_seed(M * 7 + N)
    for integer in (True, False):
        for splits in (0, 1, 3, 8):
            if integer:
                a = torch.randint(-3, 4, (M, K), generator=g).to(torch.bfloat16).to(DEV)
                w = torch.randint(-2, 3, (N, K), generator=g).to(torch.bfloat16).to(DEV)
            else:
                a = torch.randn(M, K, generator=g).to(torch.bfloat16).to(DEV)
                w = (torch.randn(N, K, generator=g) * 0.1).to(torch.bfloat16).to(DEV)
            odt = torch.float32 if (epilogue == "add" or integer) else torch.bfloat16
            out = torch.randn(M, N // 2 if epilogue == "swiglu" else N, generator=g).to(odt).to(DEV)
            ref = gemm_ref(a, w, epilogue, out)
            gemm_bf16.run("tc", out, a, w, epilogue, M, splits=splits)
            got = out.double().cpu()
            if integer and epilogue != "swiglu":
                assert torch.equal(got, ref.float().double()), (shape, splits)   # one float32 rounding
            else:
                scale = float(ref.abs().max())
                assert float((got - ref).abs().max()) <= (1e-5 if odt == torch.float32 else 1e-2) * scale
    assert gemm_bf16.status_word(torch.device(DEV)).tolist() == [0, 0, 0, 0]


@pytest.mark.parametrize("epilogue", ["store", "add", "swiglu"])
@pytest.mark.parametrize("shape", [(600, 640, 520), (512, 1000, 136), (130, 250, 192), (1100, 2560, 320),
                                   (1024, 384, 4160)])
def test_gemm_tensor_core_tokens_as_rows(shape, epilogue):
    """The orientation used for prompt-sized batches (tokens = MMA rows; a
    thread of the epilogue owns a token and writes vectors, the residual add
    leaves as reducing TMA stores where the output's pitch allows a tensor map,
    in place otherwise), with every feature tile and ragged edges, by one CTA per
    128-token tile and (-1000 - tile) by a pair of CTAs on one MMA per 256-token
    tile; the output also as a slice of a wider buffer; integer data exactly."""
    from kipp_b200.kernels import gemm_bf16
    M, N, K = shape
    g = torch.Generator().manual_seed(M + 3 * N)
    for integer in (True, False):
        for tile_f in (0, -128, -160, -192, -224, -256, -1128, -1160, -1192, -1224, -1256, -1288, -1320):
            if tile_f == 0 and M < 512:
                continue
            if integer:
                a = torch.randint(-3, 4, (M, K), generator=g).to(torch.bfloat16).to(DEV)
                w = torch.randint(-2, 3, (N, K), generator=g).to(torch.bfloat16).to(DEV)
            else:
                a = torch.randn(M, K, generator=g).to(torch.bfloat16).to(DEV)
                w = (torch.randn(N, K, generator=g) * 0.1).to(torch.bfloat16).to(DEV)
            odt = torch.float32 if (epilogue == "add" or integer) else torch.bfloat16
            n_out = N // 2 if epilogue == "swiglu" else N
            wide = torch.randn(M + 1, n_out + 8, generator=g).to(odt).to(DEV)
            out = wide[:M, 4:4 + n_out] if tile_f in (-160, -224, -1192) else wide[:M, :n_out].contiguous()
            before = wide.clone()
            ref = gemm_ref(a, w, epilogue, out)
            gemm_bf16.run("tc", out, a, w, epilogue, M, tile_f=tile_f)
            got = out.double().cpu()
            if not out.is_contiguous():                     # nothing beside the slice is touched
                after = wide.clone()
                after[:M, 4:4 + n_out] = before[:M, 4:4 + n_out]
                assert torch.equal(after, before), (shape, tile_f)
            if integer and epilogue != "swiglu":
                assert torch.equal(got, ref.float().double()), (shape, tile_f)
            else:
                scale = float(ref.abs().max())
                assert float((got - ref).abs().max()) <= (1e-5 if odt == torch.float32 else 1e-2) * scale
    assert gemm_bf16.status_word(torch.device(DEV)).tolist() == [0, 0, 0, 0]


@pytest.mark.parametrize("seed", [0, 1, 2])
def test_gemm_tensor_core_left_to_choose_its_kernel(seed):
    """Shapes drawn around every boundary of the choice of kernel and tile (tokens 1 to
    2,100, features 8 to 20,000, K 8 to 4,104, ragged in every direction), the three
    epilogues, both output types, with and without the row factors of a deferred norm:
    whatever kernel the launcher takes, the product matches the plain one."""
    from kipp_b200.kernels import gemm_bf16
    rng = random.Random(seed)
    for trial in range(40):
        M = rng.choice([1, 3, 8, 16, 17, 31, 32, 33, 40, 64, 65, 100, 128, 200, 256, 300, 400, 511, 512, 513, 700,
                        1000, 1023, 1024, 1025, 1300, 1536, 2048, 2100])
        N = rng.choice([8, 24, 128, 136, 256, 1000, 2560, 2568, 4096, 6144, 9000, 14400, 19456, 20000])
        K = rng.choice([8, 64, 72, 128, 520, 1024, 2560, 4104])
        epilogue = rng.choice(["store", "add", "swiglu"])
        g = torch.Generator(device=DEV).manual_seed(1000 * seed + trial)
        a = torch.randn(M, K, generator=g, device=DEV).to(torch.bfloat16)
        w = (torch.randn(N, K, generator=g, device=DEV) * 0.1).to(torch.bfloat16)
        odt = torch.float32 if epilogue == "add" else rng.choice([torch.float32, torch.bfloat16])
        out = torch.randn(M, N // 2 if epilogue == "swiglu" else N, generator=g, device=DEV).to(odt)
        prod = a.double() @ w.double().t()
        fold = None
        if epilogue != "add" and rng.random() < 0.4:
            ssq = torch.rand(M, 5, generator=g, device=DEV) * 30 + 1
            fold = gemm_bf16.fold_scale(ssq, 77, 1e-5)
            prod = prod * torch.rsqrt(ssq.double().sum(1) / 77 + 1e-5)[:, None]
        if epilogue == "add":
            ref = out.double() + prod
        elif epilogue == "swiglu":
            ref = prod[:, 0::2] / (1 + torch.exp(-prod[:, 0::2])) * prod[:, 1::2]
        else:
            ref = prod
        gemm_bf16.run("tc", out, a, w, epilogue, M, fold=fold)
        scale = float(ref.abs().max()) + 1e-9
        err = float((out.double() - ref).abs().max()) / scale
        assert err <= (2e-5 if odt == torch.float32 else 1e-2), (M, N, K, epilogue, odt, fold is not None, err)
    assert gemm_bf16.status_word(torch.device(DEV)).tolist() == [0, 0, 0, 0]


@pytest.mark.parametrize("wdtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("shape", [(1, 128, 64), (8, 256, 128), (17, 224, 192), (64, 992, 136), (100, 384, 2568),
                                   (300, 640, 520), (5, 2560, 1216)])
def test_gemm_folds_the_norm_around_it(shape, wdtype):
    """The few-token kernel with an RMSNorm folded in: the residual add also leaves
    bf16(new residual x norm weight) and the sums of squares of the new residual per
    32 features; a store or SwiGLU product scales row t by 1 / sqrt(sum / n + eps).
    Integer data exactly; every K split, the cluster's reduction included."""
    from kipp_b200.kernels import gemm_bf16
    M, N, K = shape
    g = torch.Generator().manual_seed(M * 5 + N)
    for splits in (0, 1, 3, 8):
        a = torch.randint(-3, 4, (M, K), generator=g).to(torch.bfloat16).to(DEV)
        w = torch.randint(-2, 3, (N, K), generator=g).to(torch.bfloat16).to(DEV)
        base = torch.randint(-8, 9, (M, N), generator=g).float().to(DEV)
        nw = (torch.randint(1, 5, (N,), generator=g).float() * 0.25).to(wdtype).to(DEV)
        out = base.clone()
        xn = torch.full((M, N + 8), 7.0, dtype=torch.bfloat16, device=DEV)
        ssq = torch.full((M, N // 32), -1.0, device=DEV)
        gemm_bf16.run("tc", out, a, w, "add", M, splits=splits, fold=gemm_bf16.fold_emit(nw, xn, ssq))
        ref = gemm_ref(a, w, "add", base).float()
        assert torch.equal(out.cpu(), ref), (shape, splits)
        assert torch.equal(xn[:, :N].float().cpu(), (ref * nw.float().cpu()).to(torch.bfloat16).float())
        assert torch.all(xn[:, N:] == 7.0)
        assert torch.equal(ssq.cpu(), (ref * ref).view(M, N // 32, 32).sum(-1))
        # the consumer: rows scaled by the factor that the sums give
        eps = 1e-3
        rstd = 1.0 / torch.sqrt(ssq.double().cpu().sum(-1, keepdim=True) / N + eps)
        for epilogue in ("store", "swiglu"):
            n_out = N // 2 if epilogue == "swiglu" else N
            got = torch.zeros(M, n_out, device=DEV)
            gemm_bf16.run("tc", got, a, w, epilogue, M, splits=splits, fold=gemm_bf16.fold_scale(ssq, N, eps))
            p = (a.double().cpu() @ w.double().cpu().t()) * rstd
            want = P.plain_silu(p[:, 0::2]) * p[:, 1::2] if epilogue == "swiglu" else p
            assert float((got.double().cpu() - want).abs().max()) <= 2e-6 * max(1.0, float(want.abs().max()))
        # ... and so do the kernels of prompt-sized batches (forced here), which cannot emit
        for tile_f in (-128, -1160):
            for epilogue in ("store", "swiglu"):
                n_out = N // 2 if epilogue == "swiglu" else N
                got = torch.zeros(M, n_out, device=DEV)
                gemm_bf16.run("tc", got, a, w, epilogue, M, tile_f=tile_f, fold=gemm_bf16.fold_scale(ssq, N, eps))
                p = (a.double().cpu() @ w.double().cpu().t()) * rstd
                want = P.plain_silu(p[:, 0::2]) * p[:, 1::2] if epilogue == "swiglu" else p
                assert float((got.double().cpu() - want).abs().max()) <= 2e-6 * max(1.0, float(want.abs().max()))
            with pytest.raises(Exception):
                gemm_bf16.run("tc", out, a, w, "add", M, tile_f=tile_f, fold=gemm_bf16.fold_emit(nw, xn, ssq))
    assert gemm_bf16.status_word(torch.device(DEV)).tolist() == [0, 0, 0, 0]


def test_gemm_refuses_what_it_cannot_take():
    from kipp_b200.kernels import KernelError, gemm_bf16
    a = torch.zeros(4, 20, dtype=torch.bfloat16, device=DEV)          # K = 20: row pitch not 16-byte
    w = torch.zeros(8, 20, dtype=torch.bfloat16, device=DEV)
    out = torch.zeros(4, 8, dtype=torch.bfloat16, device=DEV)
    assert not gemm_bf16.tc_ok(a, w)
    with pytest.raises(KernelError):
        gemm_bf16.run("tc", out, a, w, "store", 4)
    ops().gemm(out, a, w, "store")                                     # the default path takes it (CUDA cores)
    with pytest.raises(KernelError):
        ops().gemm(out, a.cpu(), w, "store")


# ------------------------------------------------------------------ norm + rotation + cache write
@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("case", [dict(D=16, nq=4, nkv=2, rot=16, norm=True, page=4),
                                  dict(D=80, nq=3, nkv=3, rot=80, norm=True, page=16),
                                  dict(D=128, nq=8, nkv=1, rot=128, norm=False, page=8),
                                  dict(D=64, nq=2, nkv=2, rot=32, norm=True, page=16),
                                  dict(D=256, nq=2, nkv=1, rot=0, norm=True, page=32),
                                  dict(D=128, nq=9, nkv=3, rot=128, norm=True, page=16, long=290),
                                  dict(D=48, nq=5, nkv=5, rot=16, norm=True, page=8, long=260),
                                  dict(D=64, nq=5, nkv=2, rot=64, norm=True, page=8, long=130, w16=True),
                                  dict(D=256, nq=3, nkv=2, rot=256, norm=True, page=16, long=70, w16=True)])
def test_qk_norm_rope_write(case, dtype):
    """Cases with `long` have many tokens: several heads per warp.  In bfloat16
    the head sizes 64, 128 and 256 with a full or no rotation take the
    16-byte-vector kernel (head counts that leave a warp's last heads empty or
    put a key and a value head into one warp); `w16` has the norm weights in
    bfloat16 as checkpoints store them."""
    D, nq, nkv, rot, page = case["D"], case["nq"], case["nkv"], case["rot"], case["page"]
    g = torch.Generator().manual_seed(D)
    n_long = case.get("long", 19)
    entries = [StepEntry("a", [0] * 5, []), StepEntry("b", [0] * 1, []), StepEntry("c", [0] * n_long, [])]
    starts = [13, 40, 0]
    width = -(-max(45, n_long + 1) // page)
    n_pages = 3 * width
    perm = torch.randperm(n_pages, generator=g).int().numpy().reshape(3, width)
    meta = pack_step(entries, starts, [0, 1, 2], [perm.astype(np.int32)], torch.device(DEV))
    T = meta.tokens
    qkv = torch.randn(T, (nq + 2 * nkv) * D, generator=g).to(dtype).to(DEV)
    wdt = torch.bfloat16 if case.get("w16") else torch.float32
    qw = (1 + 0.2 * torch.randn(D, generator=g)).to(wdt).to(DEV) if case["norm"] else None
    kw = (1 + 0.2 * torch.randn(D, generator=g)).to(wdt).to(DEV) if case["norm"] else None
    theta = 10000.0
    inv = None
    if rot:
        i = torch.arange(rot // 2, dtype=torch.float32)
        inv = torch.pow(torch.tensor(theta, dtype=torch.float64), (-(2.0 * i) / rot).double()).float().to(DEV)
    q_out = torch.zeros(T, nq, D, dtype=dtype, device=DEV)
    kp = torch.zeros(n_pages, nkv, page, D, dtype=dtype, device=DEV)
    vp = torch.zeros_like(kp)
    st = status()
    ops().qk_norm_rope_write(qkv, q_out, kp, vp, qw, kw, 1e-6, inv, rot, meta.positions,
                             meta.entry_of_token, meta.block_tables[0], page, T, nq, nkv, D, True, st)
    assert st.tolist() == [0, 0, 0, 0]
    x = qkv.double().cpu().reshape(T, nq + 2 * nkv, D)
    pos = meta.positions.cpu().tolist()

    def transform(h, w):
        if w is not None:
            h = P.plain_rmsnorm(h, w.cpu(), 1e-6)
        if rot:
            h = torch.cat([P.plain_rope(h[..., :rot].float(), pos, theta), h[..., rot:].double()], -1)
        return h
    q_ref, k_ref, v_ref = transform(x[:, :nq], qw), transform(x[:, nq:nq + nkv], kw), x[:, nq + nkv:]
    assert torch.allclose(q_out.double().cpu(), q_ref, **tol(dtype))
    ent = meta.entry_of_token.cpu().tolist()
    written = torch.zeros(n_pages, page, dtype=torch.bool)
    for t in range(T):
        pg, sl = int(perm[ent[t], pos[t] // page]), pos[t] % page
        assert torch.allclose(kp[pg, :, sl].double().cpu(), k_ref[t], **tol(dtype)), t
        assert torch.allclose(vp[pg, :, sl].double().cpu(), v_ref[t], **tol(dtype)), t
        written[pg, sl] = True
    assert float(kp.float().abs().sum(dim=(1, 3)).cpu()[~written].sum()) == 0.0    # nothing else touched
    # a run that reads another run's cache writes nothing
    kp2 = torch.zeros_like(kp)
    ops().qk_norm_rope_write(qkv, q_out, kp2, kp2, qw, kw, 1e-6, inv, rot, meta.positions,
                             meta.entry_of_token, meta.block_tables[0], page, T, nq, nkv, D, False, st)
    assert float(kp2.float().abs().sum()) == 0.0


@pytest.mark.parametrize("case", [
    dict(T=1024, nq=4, nkv=2, K=192, norm=True, rot=True, page=16, scaled=False),
    dict(T=1300, nq=5, nkv=1, K=320, norm=True, rot=True, page=8, scaled=True, w16=True),   # 7 heads: half a tile empty
    dict(T=1100, nq=2, nkv=2, K=128, norm=False, rot=True, page=64, scaled=False),
    dict(T=1030, nq=3, nkv=3, K=256, norm=True, rot=False, page=32, scaled=True),
])
def test_projection_hands_its_heads_to_attention(case):
    """The q/k/v projection of a prompt-sized step with per-head norm, rotation and
    the cache write in its epilogue: the same bits as the stored product followed
    by `qk_norm_rope_write`, with and without the row factors of a deferred norm;
    two requests in the step, permuted pages, a token count that fills no tile."""
    from kipp_b200.kernels import gemm_bf16
    D = 128
    T, nq, nkv, K, page = case["T"], case["nq"], case["nkv"], case["K"], case["page"]
    assert gemm_bf16.heads_ok(T, D, D if case["rot"] else 0) and not gemm_bf16.heads_ok(1023, D, D)
    assert not gemm_bf16.heads_ok(T, 64, 64) and not gemm_bf16.heads_ok(T, D, 64)
    g = torch.Generator().manual_seed(T + nq)
    n_a = 37
    entries = [StepEntry("a", [0] * n_a, []), StepEntry("b", [0] * (T - n_a), [])]
    starts = [29, 3]
    width = -(-(T + 40) // page)
    perm = torch.randperm(2 * width, generator=g).int().numpy().reshape(2, width)
    meta = pack_step(entries, starts, [0, 1], [perm.astype(np.int32)], torch.device(DEV))
    a = torch.randn(T, K, generator=g).to(torch.bfloat16).to(DEV)
    w = (torch.randn((nq + 2 * nkv) * D, K, generator=g) / math.sqrt(K)).to(torch.bfloat16).to(DEV)
    wdt = torch.bfloat16 if case.get("w16") else torch.float32
    qw = (1 + 0.2 * torch.randn(D, generator=g)).to(wdt).to(DEV) if case["norm"] else None
    kw = (1 + 0.2 * torch.randn(D, generator=g)).to(wdt).to(DEV) if case["norm"] else None
    inv = None
    cos_sin = by_pair = None
    if case["rot"]:
        i = torch.arange(D // 2, dtype=torch.float32)
        inv = torch.pow(torch.tensor(10000.0, dtype=torch.float64), (-(2.0 * i) / D).double()).float().to(DEV)
        cos_sin = ops().rope_table(meta.positions, inv, T)
        by_pair = ops().rope_table(meta.positions, inv, T, by_pair=True)
        assert torch.equal(by_pair.transpose(0, 1), cos_sin)
    fold = None
    if case["scaled"]:
        ssq = (torch.rand(T, 3, generator=g) * 40 + 1).to(DEV)
        fold = gemm_bf16.fold_scale(ssq, 96, 1e-5)
    st = status()

    def pools():
        return (torch.zeros(T, nq, D, dtype=torch.bfloat16, device=DEV),
                torch.zeros(2 * width, nkv, page, D, dtype=torch.bfloat16, device=DEV),
                torch.zeros(2 * width, nkv, page, D, dtype=torch.bfloat16, device=DEV))
    q1, k1, v1 = pools()
    qkv = torch.empty(T, (nq + 2 * nkv) * D, dtype=torch.bfloat16, device=DEV)
    gemm_bf16.run("tc", qkv, a, w, "store", T, fold=fold, status=st)
    ops().qk_norm_rope_write(qkv, q1, k1, v1, qw, kw, 1e-6, inv, D if case["rot"] else 0, meta.positions,
                             meta.entry_of_token, meta.block_tables[0], page, T, nq, nkv, D, True, st,
                             cos_sin=cos_sin)
    q2, k2, v2 = pools()
    gemm_bf16.run_heads(a, w, q2, k2, v2, qw, kw, 1e-6, by_pair, meta.positions, meta.entry_of_token,
                        meta.block_tables[0], nq, nkv, status=st, fold=fold)
    torch.cuda.synchronize()
    assert st.tolist() == [0, 0, 0, 0]
    assert float(q1.float().abs().sum()) > 0 and float(k1.float().abs().sum()) > 0
    assert torch.equal(q1, q2) and torch.equal(k1, k2) and torch.equal(v1, v2)
    # a run that reads another run's cache writes nothing
    q3, k3, v3 = pools()
    gemm_bf16.run_heads(a, w, q3, k3, v3, qw, kw, 1e-6, by_pair, meta.positions, meta.entry_of_token,
                        meta.block_tables[0], nq, nkv, write_cache=False, status=st, fold=fold)
    assert torch.equal(q1, q3) and float(k3.float().abs().sum()) == 0.0 and float(v3.float().abs().sum()) == 0.0
    # an unmapped page is refused through the status word and nothing is written there
    table = meta.block_tables[0].clone()
    table[1, 5] = -1
    q4, k4, v4 = pools()
    gemm_bf16.run_heads(a, w, q4, k4, v4, qw, kw, 1e-6, by_pair, meta.positions, meta.entry_of_token, table,
                        nq, nkv, status=st, fold=fold)
    assert st.tolist() == [2, 0, 0, 0]
    st.zero_()
    untouched = int(perm[1, 5])
    assert float(k4[untouched].float().abs().sum()) == 0.0
    others = [i for i in range(2 * width) if i != untouched]
    assert torch.equal(k4[others], k1[others]) and torch.equal(q4, q1)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("D", [48, 128])
def test_no_infinity_or_nan_reaches_the_cache(D, dtype):
    """A page goes from one request to the next as it is, and kernels that read whole
    tiles multiply masked keys and values by zero: so a key or value that is not
    finite (an overflow in one request) is stored as 0, in both kernels that write
    the cache."""
    nq, nkv, page, T = 4, 2, 8, 5
    g = torch.Generator().manual_seed(D)
    entries = [StepEntry("a", [0] * T, [])]
    meta = pack_step(entries, [0], [0], [np.arange(2, dtype=np.int32).reshape(1, 2)], torch.device(DEV))
    qkv = torch.randn(T, (nq + 2 * nkv) * D, generator=g).to(dtype)
    k0, v0 = nq * D, (nq + nkv) * D
    qkv[1, k0 + 3] = float("inf")              # a key element; with the norm the whole head turns NaN
    qkv[2, v0 + 5] = float("nan")
    qkv[3, v0 + D + 1] = float("-inf")
    qkv = qkv.to(DEV)
    kw = torch.ones(D, device=DEV)
    kp = torch.zeros(2, nkv, page, D, dtype=dtype, device=DEV)
    vp = torch.zeros_like(kp)
    q_out = torch.zeros(T, nq, D, dtype=dtype, device=DEV)
    st = status()
    ops().qk_norm_rope_write(qkv, q_out, kp, vp, kw, kw, 1e-6, None, 0, meta.positions, meta.entry_of_token,
                             meta.block_tables[0], page, T, nq, nkv, D, True, st)
    torch.cuda.synchronize()
    assert torch.isfinite(kp.float()).all() and torch.isfinite(vp.float()).all()
    assert float(kp[0, 0, 1].float().abs().sum()) == 0.0           # the poisoned key head became zeros
    assert float(vp[0, 0, 2, 5]) == 0.0 and float(vp[0, 1, 3, 1]) == 0.0
    assert float(vp[0, 0, 2, 4]) == float(qkv[2, v0 + 4])          # its finite neighbours are kept
    assert float(kp[0, 1, 1].float().abs().sum()) > 0              # and the other key head of that token


# ------------------------------------------------------------------ attention
def attention_case(seed, D, nq, nkv, page, layout, dtype, width=None, order="permuted"):
    """layout: list of (cached tokens, new tokens).  Random pages in a permuted
    pool (order "consecutive": page ids in a row, as a request gets them from a
    fresh pool; "runs": rows of 1 to 9 consecutive ids, in shuffled order);
    returns everything the kernels and the reference need."""
    g = torch.Generator().manual_seed(seed)
    entries = [StepEntry(i, [0] * n, []) for i, (_, n) in enumerate(layout)]
    starts = [c for c, _ in layout]
    need = [-(-(c + n) // page) for c, n in layout]
    width = width or max(need)
    n_pages = sum(need) + 3
    if order == "consecutive":
        perm = list(range(2, n_pages))
    elif order == "runs":
        runs, at = [], 0
        while at < n_pages:
            k = int(torch.randint(1, 10, (1,), generator=g))
            runs.append(list(range(at, min(at + k, n_pages))))
            at += k
        perm = [x for i in torch.randperm(len(runs), generator=g).tolist() for x in runs[i]]
    else:
        perm = torch.randperm(n_pages, generator=g).int().tolist()
    table = np.full((len(layout), width), -1, dtype=np.int32)
    at = 0
    for i, k in enumerate(need):
        table[i, :k] = perm[at:at + k]
        at += k
    meta = pack_step(entries, starts, list(range(len(layout))), [table], torch.device(DEV))
    q = torch.randn(meta.tokens, nq, D, generator=g).to(dtype).to(DEV)
    kp = torch.randn(n_pages, nkv, page, D, generator=g).to(dtype).to(DEV)
    vp = torch.randn(n_pages, nkv, page, D, generator=g).to(dtype).to(DEV)
    return meta, table, q, kp, vp


def attention_ref(meta, table, q, kp, vp, layout, page, window, scale):
    T, nq, D = q.shape
    nkv = kp.shape[1]
    out = torch.zeros(T, nq, D, dtype=torch.float64)
    qc, kc, vc = q.double().cpu(), kp.double().cpu(), vp.double().cpu()
    t = 0
    for e, (ctx, n) in enumerate(layout):
        total = ctx + n
        pages = torch.tensor(table[e, :-(-total // page)].tolist())
        keys = kc[pages].permute(0, 2, 1, 3).reshape(-1, nkv, D)[:total]
        vals = vc[pages].permute(0, 2, 1, 3).reshape(-1, nkv, D)[:total]
        for i in range(n):
            pos = ctx + i
            lo = 0 if not window else max(0, pos - window + 1)
            for h in range(nq):
                gk = h // (nq // nkv)
                s = (keys[lo:pos + 1, gk] @ qc[t, h]) * scale
                out[t, h] = P.plain_softmax(s) @ vals[lo:pos + 1, gk]
            t += 1
    return out


LAYOUTS = [[(0, 70), (130, 1), (5, 2), (63, 66), (300, 1)],
           [(0, 1), (1, 1), (15, 1), (16, 1), (255, 1), (256, 1), (257, 1), (700, 1)],
           [(0, 200)], [(100, 3), (0, 64), (64, 64), (127, 2)]]


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("window", [None, 37])
@pytest.mark.parametrize("shape", [dict(D=16, nq=4, nkv=2, page=16), dict(D=48, nq=6, nkv=3, page=8),
                                   dict(D=128, nq=8, nkv=1, page=4), dict(D=256, nq=2, nkv=2, page=32),
                                   dict(D=20, nq=10, nkv=1, page=16), dict(D=7, nq=3, nkv=1, page=8)])
def test_attention_simt(shape, window, dtype):
    D, nq, nkv, page = shape["D"], shape["nq"], shape["nkv"], shape["page"]
    for li, layout in enumerate(LAYOUTS[:2] + LAYOUTS[3:]):
        meta, table, q, kp, vp = attention_case(li, D, nq, nkv, page, layout, dtype)
        out = torch.zeros_like(q)
        st = status()
        ops().attention(out, q, kp, vp, meta, meta.block_tables[0], page, nq, nkv, D, 1 / math.sqrt(D),
                        window, st, impl="simt")
        ref = attention_ref(meta, table, q, kp, vp, layout, page, window, 1 / math.sqrt(D))
        assert st.tolist() == [0, 0, 0, 0]
        assert torch.allclose(out.double().cpu(), ref, **tol(dtype)), (shape, li)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("shape", [dict(D=256, nq=2, nkv=2, page=16), dict(D=72, nq=9, nkv=3, page=8), dict(D=30, nq=4, nkv=2, page=4)])
def test_attention_simt_stages(shape, dtype):
    """Few blocks have two tiles of keys on their way, many one: a token's result has the same bits among 6 and among
    4,800, in rows of whole 16-byte pieces and others, with a window that begins inside a tile."""
    D, nq, nkv, page = shape["D"], shape["nq"], shape["nkv"], shape["page"]
    few, times = [(0, 1), (31, 1), (32, 2), (100, 1), (130, 1)], 800
    for window in (None, 40):
        meta, table, q, kp, vp = attention_case(3, D, nq, nkv, page, few, dtype)
        out, st = torch.zeros_like(q), status()
        run = lambda o, x, m: ops().attention(o, x, kp, vp, m, meta.block_tables[0], page, nq, nkv, D, 1 / math.sqrt(D), window, st, impl="simt")   # noqa: E731
        run(out, q, meta)
        ref = attention_ref(meta, table, q, kp, vp, few, page, window, 1 / math.sqrt(D))
        assert torch.allclose(out.double().cpu(), ref, **tol(dtype))
        class Many:
            tokens = meta.tokens * times
            positions, entry_of_token = meta.positions[:meta.tokens].repeat(times), meta.entry_of_token[:meta.tokens].repeat(times)
        among = torch.zeros(Many.tokens, nq, D, dtype=dtype, device=DEV)
        run(among, q.repeat(times, 1, 1), Many)
        assert torch.equal(among, out.repeat(times, 1, 1)) and st.tolist() == [0, 0, 0, 0]


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("shape", [dict(D=128, nq=16, nkv=2, page=16), dict(D=128, nq=4, nkv=1, page=8), dict(D=64, nq=2, nkv=2, page=16),
                                   dict(D=40, nq=12, nkv=1, page=32), dict(D=128, nq=9, nkv=3, page=4)])
def test_attention_simt_of_few_blocks(shape, dtype):
    """A block for each SM at most: four tiles of keys at a time.  Contexts that end inside the first tile, at the ends of
    tiles and of four of them, and windows that begin inside each: the bits that a token has among thousands, where
    the tiles go one by one."""
    D, nq, nkv, page = shape["D"], shape["nq"], shape["nkv"], shape["page"]
    few, times = [(0, 1), (31, 1), (126, 3), (255, 2), (400, 1)], 500
    for window in (None, 33, 150):
        meta, table, q, kp, vp = attention_case(5, D, nq, nkv, page, few, dtype)
        out, st = torch.zeros_like(q), status()
        run = lambda o, x, m: ops().attention(o, x, kp, vp, m, meta.block_tables[0], page, nq, nkv, D, 1 / math.sqrt(D), window, st, impl="simt")   # noqa: E731
        run(out, q, meta)
        ref = attention_ref(meta, table, q, kp, vp, few, page, window, 1 / math.sqrt(D))
        assert torch.allclose(out.double().cpu(), ref, **tol(dtype))
        class Many:
            tokens = meta.tokens * times
            positions, entry_of_token = meta.positions[:meta.tokens].repeat(times), meta.entry_of_token[:meta.tokens].repeat(times)
        among = torch.zeros(Many.tokens, nq, D, dtype=dtype, device=DEV)
        run(among, q.repeat(times, 1, 1), Many)
        assert torch.equal(among, out.repeat(times, 1, 1)) and st.tolist() == [0, 0, 0, 0]


@pytest.mark.parametrize("dtype", DTYPES)
def test_attention_simt_before_the_first_visible_key(dtype):
    """Tiles of keys whose scores are all -inf count for nothing before a score that is not, whatever their values: infinite ones do not
    reach a result, neither where four tiles go at a time (few blocks) nor one by one.  They end with a tile, with
    four of them, or with the context, and the result is then 0."""
    D, nq, nkv, page = 128, 8, 2, 16
    contexts, gone = [300, 170, 140, 31, 127, 200], [64, 128, 32, 32, 128, 201]          # a context's first keys score -inf
    meta, table, q, kp, vp = attention_case(9, D, nq, nkv, page, [(c, 1) for c in contexts], dtype)
    q = q.abs() + 0.5
    for e, n in enumerate(gone):
        for j in range(n):
            at = int(table[e, j // page])
            kp[at, :, j % page] = -3e38                                        # (the dot product overflows)
            vp[at, :, j % page] = float("inf")
    run = lambda o, x, m: ops().attention(o, x, kp, vp, m, meta.block_tables[0], page, nq, nkv, D, 1 / math.sqrt(D), None, status(), impl="simt")   # noqa: E731
    few, times = torch.full_like(q, 7.0), 100
    run(few, q, meta)
    class Many:
        tokens = meta.tokens * times
        positions, entry_of_token = meta.positions[:meta.tokens].repeat(times), meta.entry_of_token[:meta.tokens].repeat(times)
    among = torch.full((Many.tokens, nq, D), 7.0, dtype=dtype, device=DEV)
    run(among, q.repeat(times, 1, 1), Many)
    assert torch.isfinite(few.float()).all() and few[:3].any(dim=2).all() and not few[3:].any()
    assert torch.equal(among, few.repeat(times, 1, 1))


@pytest.mark.parametrize("asked,of_step", [(1, False), (5, False), (40, False), (40, True)])
def test_attention_simt_behind_the_cache_write(asked, of_step):
    """Attention right behind the kernel that writes the keys and values: of the last of the tokens written (the general
    entry, which waits for all of them), and of all of them beside a context that was there (a step's entry)."""
    import ctypes
    from kipp_b200.csrc.build import load_library
    D, nq, nkv, page, scale = 64, 4, 2, 16, 1 / math.sqrt(64)
    layout = [(100 if of_step else 0, 40)]
    meta, table, _, kp, vp = attention_case(4, D, nq, nkv, page, layout, torch.float32)
    g = torch.Generator().manual_seed(asked)
    name = "kipp_paged_attention_simt" + ("_of_step" if of_step else "")
    fn = getattr(load_library("attention_simt"), name)
    p, i, f = ctypes.c_void_p, ctypes.c_int, ctypes.c_float
    fn.argtypes = [p, p, p, p, i, p, p, p, i, i, i, i, i, i, f, i, p, p]
    bt, positions, entry = meta.block_tables[0], meta.positions[40 - asked:40].contiguous(), meta.entry_of_token[40 - asked:40].contiguous()
    for _ in range(10):
        qkv = torch.randn(40, (nq + 2 * nkv) * D, generator=g).to(DEV)
        q, out, st = torch.zeros(40, nq, D, device=DEV), torch.zeros(asked, nq, D, device=DEV), status()
        torch.cuda.synchronize()
        ops().qk_norm_rope_write(qkv, q, kp, vp, None, None, 1e-6, None, 0, meta.positions, meta.entry_of_token, bt, page, 40, nq, nkv, D, True, st)
        rc = fn(out.data_ptr(), q[40 - asked:].data_ptr(), kp.data_ptr(), vp.data_ptr(), 0, positions.data_ptr(), entry.data_ptr(), bt.data_ptr(),
                bt.shape[1], page, asked, nq, nkv, D, scale, 0, st.data_ptr(), torch.cuda.current_stream().cuda_stream)
        ref = attention_ref(meta, table, q, kp, vp, layout, page, None, scale)[40 - asked:]
        assert rc == 0 and st.tolist() == [0, 0, 0, 0] and torch.allclose(out.double().cpu(), ref, **tol(torch.float32))


@pytest.mark.parametrize("window", [None, 37, 300])
@pytest.mark.parametrize("shape", [dict(D=64, nq=4, nkv=2, page=16), dict(D=128, nq=8, nkv=2, page=16),
                                   dict(D=128, nq=16, nkv=1, page=8), dict(D=64, nq=3, nkv=3, page=32),
                                   dict(D=128, nq=40, nkv=2, page=16), dict(D=128, nq=4, nkv=2, page=64),
                                   dict(D=64, nq=2, nkv=1, page=128), dict(D=128, nq=2, nkv=2, page=4)])
def test_attention_tensor_core(shape, window):
    """Prompt portions and single decoded tokens through the tensor-core kernels:
    portions of 64 tokens and more through tcgen05, shorter ones and decoded
    tokens through mma.sync (a group of 20 > 16 and a page of 4 slots go through
    the mma.sync portion kernel throughout; pages of 64 and 128 slots hold a whole
    key tile); then the same with tcgen05 off."""
    from kipp_b200.kernels import attention_bf16
    D, nq, nkv, page = shape["D"], shape["nq"], shape["nkv"], shape["page"]
    assert attention_bf16.supported(D, nq, nkv)
    for li, layout in enumerate(LAYOUTS):
        meta, table, q, kp, vp = attention_case(10 + li, D, nq, nkv, page, layout, torch.bfloat16)
        out = torch.full_like(q, 9.0)
        st = status()
        # whatever lies in the split-K scratch must not matter: a split wholly behind a
        # window writes no partial output, and 0 x NaN would be NaN
        attention_bf16.decode_scratch(torch.device(DEV), meta.tokens, nq, D).fill_(float("nan"))
        ops().attention(out, q, kp, vp, meta, meta.block_tables[0], page, nq, nkv, D, 1 / math.sqrt(D),
                        window, st, impl="mma")
        ref = attention_ref(meta, table, q, kp, vp, layout, page, window, 1 / math.sqrt(D))
        assert torch.allclose(out.double().cpu(), ref, rtol=2e-2, atol=2e-2), (shape, li, window)
        assert st.tolist() == [0, 0, 0, 0]
        # the decoded tokens cut into splits of a given length instead of dealt out as a stream
        out1 = torch.full_like(q, 9.0)
        attention_bf16.run("mma", out1, q, kp, vp, meta, meta.block_tables[0], page, nq, nkv, D, 1 / math.sqrt(D),
                           window, st, stream=False)
        assert torch.allclose(out1.double().cpu(), ref, rtol=2e-2, atol=2e-2), (shape, li, window)
        attention_bf16.PREFILL_TC = False
        try:
            out2 = torch.full_like(q, 9.0)
            ops().attention(out2, q, kp, vp, meta, meta.block_tables[0], page, nq, nkv, D, 1 / math.sqrt(D),
                            window, st, impl="mma")
        finally:
            attention_bf16.PREFILL_TC = True
        assert torch.allclose(out2.double().cpu(), ref, rtol=2e-2, atol=2e-2), (shape, li, window)


@pytest.mark.parametrize("order", ["consecutive", "runs"])
@pytest.mark.parametrize("page", [8, 16, 32])
@pytest.mark.parametrize("D", [64, 128])
def test_attention_pages_in_a_row(D, page, order):
    """Pages that follow one another in the pool (what a request gets from a fresh
    pool) are fetched as whole key tiles by the prompt kernel, pages in any other
    order one by one: both in one launch, rows of consecutive pages that start and
    end anywhere in a tile."""
    nq, nkv = 4, 2
    for window in (None, 150):
        for li, layout in enumerate([[(0, 700)], [(300, 150), (0, 64), (77, 513)], [(64, 200), (1000, 129)]]):
            meta, table, q, kp, vp = attention_case(40 + li, D, nq, nkv, page, layout, torch.bfloat16, order=order)
            out = torch.full_like(q, 9.0)
            st = status()
            ops().attention(out, q, kp, vp, meta, meta.block_tables[0], page, nq, nkv, D, 1 / math.sqrt(D),
                            window, st, impl="mma")
            ref = attention_ref(meta, table, q, kp, vp, layout, page, window, 1 / math.sqrt(D))
            assert st.tolist() == [0, 0, 0, 0]
            assert torch.allclose(out.double().cpu(), ref, rtol=2e-2, atol=2e-2), (D, page, order, li, window)


@pytest.mark.parametrize("impl,dtype", [("simt", torch.float32), ("simt", torch.bfloat16),
                                        ("mma", torch.bfloat16)])
def test_attention_finds_one_far_key(impl, dtype):
    """Random data would hide a wrong key among hundreds: here each query's
    score is large for exactly one chosen key (the first key, page edges, the
    window's edge, the token itself) and the values name their position."""
    D, nq, nkv, page, window = 128, 4, 2, 16, 100      # D > the longest portion: key directions stay unique
    ctx, n = 419, 5                                  # a portion of 5 tokens, one decoded token, a portion of 70
    for layout in ([(ctx, n)], [(ctx + n - 1, 1)], [(ctx, 70)]):
        meta, table, q, kp, vp = attention_case(3, D, nq, nkv, page, layout, dtype)
        total = layout[0][0] + layout[0][1]
        kp.zero_(); vp.zero_(); q.zero_()
        pages = table[0]
        for pos in range(total):                     # key at pos: e_{pos % D} scaled; value: its position
            kp[pages[pos // page], :, pos % page, pos % D] = 1.0
            vp[pages[pos // page], :, pos % page, 0] = float(pos % 256)
            vp[pages[pos // page], :, pos % page, 1] = float(pos // 256)
        first = layout[0][0]                          # position of the first query
        for win, targets in ((None, [0, 15, 16, 255, 256, first - 65, first - 1, "self"]),
                             (window, ["edge", "edge+1", "mid", "self"])):
            for target in targets:
                q.zero_()
                want = []
                for i in range(layout[0][1]):
                    pos = layout[0][0] + i
                    j = {"self": pos, "edge": pos - window + 1, "edge+1": pos - window + 2,
                         "mid": pos - window // 2}.get(target, target)
                    q[i, :, j % D] = 60.0
                    want.append(j)
                # keys j + k * D point the same way as key j: the wanted key alone is twice as long
                for i, j in enumerate(want):
                    kp[pages[j // page], :, j % page, j % D] = 2.0
                out = torch.zeros_like(q)
                ops().attention(out, q, kp, vp, meta, meta.block_tables[0], page, nq, nkv, D, 1.0, win,
                                status(), impl=impl)
                got = out.float().cpu()
                for i, j in enumerate(want):
                    pos_read = got[i, :, 0] + 256 * got[i, :, 1]
                    assert torch.allclose(pos_read, torch.full((nq,), float(j)), atol=0.6), (target, i, j, pos_read)
                for j in want:
                    kp[pages[j // page], :, j % page, j % D] = 1.0
        # a key just outside the window must NOT be seen even when it is the strongest
        q.zero_()
        pos = layout[0][0] + layout[0][1] - 1
        j = pos - window                               # one before the window's first key
        q[-1, :, j % D] = 60.0
        kp[pages[j // page], :, j % page, j % D] = 4.0
        out = torch.zeros_like(q)
        ops().attention(out, q, kp, vp, meta, meta.block_tables[0], page, nq, nkv, D, 1.0, window, status(),
                        impl=impl)
        got = out.float().cpu()[-1]
        assert (got[:, 0] + 256 * got[:, 1] - float(j)).abs().min() > 1.0
        kp[pages[j // page], :, j % page, j % D] = 1.0


@pytest.mark.parametrize("rate", [0.02, 0.07, 0.3, -0.07])
def test_attention_scores_that_climb(rate):
    """Scores that rise (or fall) steadily with the key's position: the running
    maximum of the prompt kernel drifts by a few units per key tile, so tiles are
    added under a maximum that is not their own before the output is rescaled;
    with random scores the maximum settles in the first tiles and this path sleeps."""
    D, nq, nkv, page = 128, 4, 2, 16
    for layout in ([(0, 700)], [(300, 150), (0, 64)]):
        meta, table, q, kp, vp = attention_case(21, D, nq, nkv, page, layout, torch.bfloat16)
        kp.mul_(0.1)
        q.mul_(0.1)
        q[:, :, 5] = 1.0
        for r, (ctx, n) in enumerate(layout):
            for pos in range(ctx + n):
                kp[table[r][pos // page], :, pos % page, 5] = rate * pos      # score = rate * pos in natural-log units
        out = torch.zeros_like(q)
        st = status()
        ops().attention(out, q, kp, vp, meta, meta.block_tables[0], page, nq, nkv, D, 1.0, None, st, impl="mma")
        ref = attention_ref(meta, table, q, kp, vp, layout, page, None, 1.0)
        assert st.tolist() == [0, 0, 0, 0]
        assert torch.allclose(out.double().cpu(), ref, rtol=2e-2, atol=2e-2), (rate, layout)


# ------------------------------------------------------------------ sampling
def test_burst_advance_moves_a_step_on():
    """The kernels between two greedy steps of a burst: tokens handed over and put into
    the ring row the counter names, positions and cached lengths + 1; then the keys per
    decode-attention split of every token, chosen as the host chooses them for the new
    lengths (for the whole step, or from each token's own context)."""
    from kipp_b200.kernels import attention_bf16, sampling
    g = torch.Generator().manual_seed(5)
    for n, longest in ((1, 100), (1, 2047), (3, 5000), (8, 8190), (8, 127), (64, 2047), (64, 40_000), (130, 700)):
        lens = torch.randint(1, longest + 1, (n,), generator=g).int()
        lens[int(torch.randint(0, n, (1,), generator=g))] = longest
        dev = lambda t: t.clone().to(DEV)
        tokens, positions, context = dev(torch.zeros(n).int()), dev(lens), dev(lens)
        counter = dev(torch.tensor([2]).int())
        nxt = torch.randint(0, 50_000, (n,), generator=g).int()
        ring = torch.full((4, n), -7, dtype=torch.int32, device=DEV)
        sampling.burst_advance(tokens, positions, context, dev(nxt), ring, counter)
        assert tokens.cpu().tolist() == nxt.tolist()
        assert positions.cpu().tolist() == (lens + 1).tolist() == context.cpu().tolist()
        assert int(counter) == 3 and ring[2].cpu().tolist() == nxt.tolist()
        assert ring[[0, 1, 3]].eq(-7).all()
        # the next step's tokens sit at positions lens + 1 and see lens + 2 keys
        rows = dev(torch.arange(n).int())
        split = dev(torch.zeros(n + 3).int())
        for kv_heads, sms in ((8, 148), (2, 148), (1, 132)):
            attention_bf16.decode_replan(split, context, rows, kv_heads, 3 * sms, 5, 32, own_length=False)
            want = split_length(n, longest + 2, kv_heads, sms)
            assert split[:n].cpu().tolist() == [want] * n, (n, longest, kv_heads)
            assert split[n:].eq(0).all()
        attention_bf16.decode_replan(split, context, rows, 8, 444, 5, 32, own_length=True)
        assert split[:n].cpu().tolist() == [split_length(1, int(x) + 2, own=True) for x in lens]
        # a full ring: the tokens are still handed over, no row is written
        counter.fill_(4)
        sampling.burst_advance(tokens, positions, context, dev(nxt), ring, counter)
        assert int(counter) == 5 and ring[[0, 1, 3]].eq(-7).all()


@pytest.mark.parametrize("n", [1000, 8191, 8192, 151936, 300001])
def test_argmax_first_maximum(n):
    """Short rows by one block, long rows shared among blocks: the first maximum either way,
    also where the maxima sit in different shares, and index 0 for a row without a number."""
    logits = torch.randn(7, n + 3, generator=torch.Generator().manual_seed(1))[:, :n].to(DEV)     # a pitch beside n
    logits[1, 7] = logits[1, n - 100] = 50.0
    logits[2, :] = 0.25
    logits[5, :] = float("nan")
    logits[6, :] = float("-inf")
    logits[6, : n // 2] = float("nan")
    out = ops().argmax_rows(logits).cpu().tolist()
    assert out == [int(logits[0].argmax()), 7, 0, int(logits[3].argmax()), int(logits[4].argmax()), 0, n // 2]


@pytest.mark.parametrize("vocab", [1000, 151936])
def test_sample_rows_draws_the_plain_sampler_tokens(vocab):
    from kipp_b200.kernels import sampling as ks
    g = torch.Generator().manual_seed(vocab)
    cases = [dict(temperature=0.0), dict(temperature=0.8), dict(temperature=1.3, top_k=5),
             dict(temperature=0.7, top_p=0.6), dict(temperature=1.0, min_p=0.2),
             dict(temperature=0.9, top_k=40, top_p=0.9, min_p=0.02), dict(temperature=0.25),
             dict(temperature=5.0, top_p=0.95), dict(temperature=1.0, top_k=1), dict(temperature=2.0, top_k=vocab + 5)]
    rows = len(cases)
    logits = (torch.randn(rows, vocab, generator=g) * 2.5)
    logits[:, 17] = logits[:, 200] = logits.max(dim=1).values - 0.25       # ties inside the candidates
    dev = logits.to(DEV)
    state = 99
    for trial in range(12):
        uni, want = [], []
        for r, c in enumerate(cases):
            tok, new_state = P.plain_sample(logits[r].numpy(), rng_state=state + r, **{"temperature": 0.0, **c})
            _, u = P.uniform_unit(state + r)
            uni.append(u)
            want.append(tok)
        f = lambda key, default, dt: torch.tensor([c.get(key, default) for c in cases], dtype=dt, device=DEV)
        got = ks.sample_rows(dev, f("temperature", 0.0, torch.float32), f("top_k", 0, torch.int32),
                             f("top_p", 1.0, torch.float32), f("min_p", 0.0, torch.float32),
                             torch.tensor(uni, dtype=torch.float64, device=DEV)).cpu().tolist()
        assert got == want, (trial, got, want)
        state = state * 7 + 13


def test_sample_rows_with_buckets_longer_than_a_blocks_list():
    """Rows whose candidates share one value or a few (more than the 4,096 that a block lists, so the passes
    after the first go over the whole row again), a top-k just under, at and above that number, and a set that empties
    but for its first: the tokens of the plain sampler."""
    from kipp_b200.kernels import sampling as ks
    n = 40000
    logits = torch.zeros(6, n)
    logits[1, ::2] = 1e-7                                       # two values a rounding apart
    logits[2] = torch.arange(n) % 3 * 0.5
    logits[3:] = torch.randn(3, n, generator=torch.Generator().manual_seed(3)) * 1e-3
    k = [0, 9000, 0, 4095, 4096, 4097]
    top_p, min_p = [0.7, 1.0, 0.3, 0.9, 1.0, 0.9], [0.0, 0.0, 1.0, 0.0, 0.5, 0.0]
    for u in (0.0, 0.3, 0.999):
        want = []
        for r in range(6):
            # the uniform number comes from the state's first draw: look for the token by its definition instead
            order = np.lexsort((np.arange(n), -logits[r].numpy().astype(np.float64)))
            order = order[: k[r] or n]
            w = np.exp((logits[r].numpy()[order] - logits[r].numpy()[order[0]]).astype(np.float32)).astype(np.float64)
            keep = w >= min_p[r]
            order, w = order[keep], w[keep]
            c = np.cumsum(w)
            last = int(np.searchsorted(c, top_p[r] * c[-1])) if top_p[r] < 1 else len(w) - 1
            want.append((order, c, u * c[min(last, len(w) - 1)]))
        got = ks.sample_rows(logits.to(DEV), torch.ones(6, device=DEV), torch.tensor(k, dtype=torch.int32, device=DEV),
                             torch.tensor(top_p, device=DEV), torch.tensor(min_p, device=DEV),
                             torch.full((6,), u, dtype=torch.float64, device=DEV)).cpu().tolist()
        for r, (order, c, draw) in enumerate(want):
            # the running sums of 40,000 weights are exact to 2^-23 of their unit: the token or its neighbour
            at = int(np.nonzero(order == got[r])[0][0])
            assert c[at] >= draw - 1e-2 and (at == 0 or c[at - 1] <= draw + 1e-2), (u, r, got[r])


@pytest.mark.parametrize("vocab", [8188, 8192, 8195, 65537, 131040, 131044, 262200])
def test_sample_rows_alone_and_among_others(vocab):
    """Long parts of a row are counted in a histogram for each lane, 131,040 elements at a time, short ones by groups of equal
    buckets: a row's token is the same whether eight blocks share it or one walks it among 80, on both sides of either limit."""
    from kipp_b200.kernels import sampling as ks
    rows, some = 80, 8
    g = torch.Generator().manual_seed(vocab)
    logits = torch.randn(some, vocab, generator=g) * torch.tensor([0.1, 1.0, 3.0, 10.0, 0.01, 2.0, 1.0, 5.0])[:, None]
    logits[6, ::3] = 0.5
    k = torch.tensor([0, 0, 50, 0, 5000, 0, 0, 0], dtype=torch.int32)
    p = torch.tensor([0.95, 1.0, 0.9, 0.5, 0.99, 0.3, 0.7, 0.9999])
    mp = torch.tensor([0.0, 0.0, 0.0, 0.01, 0.0, 0.2, 0.0, 0.0])
    u = torch.rand(some, generator=g, dtype=torch.float64)
    one = lambda t, n: t.repeat(n, *[1] * (t.dim() - 1)).to(DEV)                     # noqa: E731
    draw = lambda n: ks.sample_rows(one(logits, n), torch.full((some * n,), 0.8, device=DEV), one(k, n), one(p, n), one(mp, n), one(u, n))  # noqa: E731
    alone = draw(1).cpu()
    assert draw(rows // some).cpu().equal(alone.repeat(rows // some))


@pytest.mark.parametrize("rows,vocab", [(1, 151936), (80, 32000), (3, 8192)])
def test_sample_rows_of_either_form(rows, vocab):
    """A row's token is the same whether the caller says that every row has a top-k (no histograms by lane) or not, greedy rows
    among them."""
    import ctypes
    from kipp_b200.csrc.build import load_library
    fn = load_library("sampling").kipp_sample_rows_of
    p, i, ll = ctypes.c_void_p, ctypes.c_int, ctypes.c_longlong
    fn.argtypes = [p, ll, i, i, p, p, p, p, p, i, p, p]
    g = torch.Generator().manual_seed(rows)
    logits = (torch.randn(rows, vocab, generator=g) * 2).to(DEV)
    t = torch.full((rows,), 0.9, device=DEV)
    t[2::5] = 0
    k = (torch.arange(rows) * 613 % 4096 + 1).int().to(DEV)
    tp, mp = torch.rand(rows, generator=g).clamp(0.05, 1).to(DEV), (torch.rand(rows, generator=g) * 0.01).to(DEV)
    u = torch.rand(rows, generator=g, dtype=torch.float64).to(DEV)
    tokens = []
    for largest in (0, 4096):
        out = torch.full((rows,), -1, dtype=torch.int32, device=DEV)
        assert fn(logits.data_ptr(), vocab, rows, vocab, t.data_ptr(), k.data_ptr(), tp.data_ptr(), mp.data_ptr(), u.data_ptr(), largest,
                  out.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0
        tokens.append(out)
    assert torch.equal(*tokens) and tokens[0].min() >= 0 and tokens[0].max() < vocab
    assert torch.equal(tokens[0][2::5].long(), logits[2::5].argmax(dim=1))


@pytest.mark.parametrize("vocab", [700, 151936])
def test_sample_rows_at_the_ends_of_a_nucleus(vocab):
    """The draw takes its first pass from the selection that found the nucleus: 0 gives the nucleus's first token and the
    largest number below 1 its last, never one behind it, with and without top-k and min-p, where the nucleus ends in the
    first bucket of values, in a later one or with the set."""
    from kipp_b200.kernels import sampling as ks
    g = torch.Generator().manual_seed(vocab)
    cases = [(0, 0.02, 0.0), (0, 0.5, 0.0), (0, 0.9999, 0.0), (50, 0.6, 0.0), (0, 0.7, 0.3), (300, 0.99, 0.01), (1, 0.5, 0.0)]
    rows = len(cases)
    logits = torch.randn(rows, vocab, generator=g) * 2.5
    logits[:, 100:104] += 12.0                                                       # few tokens with most of the weight
    logits[1, 100:104] -= 12.0
    last, first = [], []
    for r, (k, p, mp) in enumerate(cases):
        v = logits[r].numpy()
        order = np.lexsort((np.arange(vocab), -v.astype(np.float64)))[: k or vocab]
        w = np.exp((v[order] - v[order[0]]).astype(np.float32)).astype(np.float64)
        order, w = order[(w >= mp) & (v[order] >= v[order[0]] - 20)], w[(w >= mp) & (v[order] >= v[order[0]] - 20)]
        c = np.cumsum(w)
        at = min(int(np.searchsorted(c, np.float64(np.float32(p)) * c[-1])), len(w) - 1)
        # sums are exact to 2^-23 of the top weight each: the tokens whose inclusive sums lie that near the boundary
        slack = len(w) * 2.0 ** -22
        last.append(set(order[(c >= c[at] - w[at] - slack - 1e-9) & (c - w <= c[at] + slack)].tolist()) if slack > w[at] else {int(order[at])})
        first.append(int(order[0]))
    f = lambda j, dt: torch.tensor([c[j] for c in cases], dtype=dt, device=DEV)      # noqa: E731
    for u in (0.0, 1.0 - 2.0 ** -53):
        got = ks.sample_rows(logits.to(DEV), torch.ones(rows, device=DEV), f(0, torch.int32), f(1, torch.float32), f(2, torch.float32),
                             torch.full((rows,), u, dtype=torch.float64, device=DEV)).cpu().tolist()
        for r in range(rows):
            assert got[r] == first[r] if u == 0.0 else got[r] in last[r], (u, r, got[r])


def test_penalties_and_bias_match_the_reference_sampler():
    import json
    import os
    with open(os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "operators.json")) as f:
        gold = json.load(f)["penalties"]
    from kipp_b200.kernels import sampling as ks
    logits = torch.tensor([gold["logits"], gold["logits"]], dtype=torch.float32, device=DEV)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)          # noqa: E731
    f32 = lambda v: torch.tensor(v, dtype=torch.float32, device=DEV)        # noqa: E731
    recent = gold["recent"]
    bias = {int(k): v for k, v in gold["bias"].items()}
    # row 0 has the penalties and the bias, row 1 none
    ks.apply_penalties(logits, i32([recent, [-1] * len(recent)]), i32([len(recent), 0]),
                       f32([gold["repetition"], 1.0]), f32([gold["presence"], 0.0]), f32([gold["frequency"], 0.0]),
                       i32([list(bias), [0] * len(bias)]), f32([list(bias.values()), [0.0] * len(bias)]),
                       i32([len(bias), 0]))
    out = ks.argmax_rows(logits).cpu().tolist()
    assert out[0] == gold["token"]                       # what kipp_sample_ex chose with the same settings
    assert out[1] == int(np.argmax(np.asarray(gold["logits"], dtype=np.float32))) and out[0] != out[1]


@pytest.mark.parametrize("case", [dict(D=128, nq=8, nkv=2, page=16, rot=True, norm=True, w16=True, window=None),
                                  dict(D=64, nq=6, nkv=3, page=8, rot=True, norm=True, w16=False, window=90),
                                  dict(D=128, nq=5, nkv=1, page=32, rot=False, norm=True, w16=True, window=None),
                                  dict(D=64, nq=16, nkv=1, page=16, rot=True, norm=False, w16=False, window=None)])
def test_decode_attention_fused_with_norm_rotation_and_cache_write(case):
    """A step of decoded tokens: the attention kernel that normalises, rotates and
    writes the new key and value itself against the two separate launches, on
    the same raw projection output; outputs and caches must agree (the norm's
    sum runs in another order: rounding only), and a run that does not write
    its cache leaves the pages alone."""
    from kipp_b200.kernels import attention_bf16
    D, nq, nkv, page, window = case["D"], case["nq"], case["nkv"], case["page"], case["window"]
    layout = [(700, 1), (15, 1), (16, 1), (255, 1), (1023, 1), (0, 1), (129, 1)]
    meta, table, _, kp, vp = attention_case(77, D, nq, nkv, page, layout, torch.bfloat16)
    T = meta.tokens
    g = torch.Generator().manual_seed(5)
    qkv = torch.randn(T, (nq + 2 * nkv) * D, generator=g).to(torch.bfloat16).to(DEV)
    wdt = torch.bfloat16 if case["w16"] else torch.float32
    qw = (1 + 0.2 * torch.randn(D, generator=g)).to(wdt).to(DEV) if case["norm"] else None
    kw = (1 + 0.2 * torch.randn(D, generator=g)).to(wdt).to(DEV) if case["norm"] else None
    rot = D if case["rot"] else 0
    inv = cos_sin = None
    if rot:
        i = torch.arange(D // 2, dtype=torch.float32)
        inv = torch.pow(torch.tensor(1e4, dtype=torch.float64), (-(2.0 * i) / D).double()).float().to(DEV)
        cos_sin = ops().rope_table(meta.positions, inv, T)
    assert attention_bf16.decode_fused_ok(meta, torch.bfloat16, nq, nkv, D, rot)
    st = status()
    # separate launches
    k1, v1 = kp.clone(), vp.clone()
    q = torch.zeros(T, nq, D, dtype=torch.bfloat16, device=DEV)
    ops().qk_norm_rope_write(qkv, q, k1, v1, qw, kw, 1e-6, inv, rot, meta.positions, meta.entry_of_token,
                             meta.block_tables[0], page, T, nq, nkv, D, True, st, cos_sin=cos_sin)
    want = torch.zeros_like(q)
    ops().attention(want, q, k1, v1, meta, meta.block_tables[0], page, nq, nkv, D, 1 / math.sqrt(D), window, st,
                    impl="mma")
    # one launch
    k2, v2 = kp.clone(), vp.clone()
    got = torch.full_like(q, 7.0)
    attention_bf16.decode_scratch(torch.device(DEV), T, nq, D).fill_(float("nan"))
    ops().attention_decode_fused(got, qkv, k2, v2, qw, kw, 1e-6, cos_sin, True, meta, meta.block_tables[0], page,
                                 nq, nkv, D, 1 / math.sqrt(D), window, st)
    assert st.tolist() == [0, 0, 0, 0]
    assert torch.equal(v1, v2)
    assert torch.allclose(k1.float(), k2.float(), rtol=1e-2, atol=1e-2)
    assert float((k1.float() - kp.float()).abs().sum()) > 0          # keys were written
    assert torch.allclose(got.float(), want.float(), rtol=2e-2, atol=2e-2)
    k4, v4 = kp.clone(), vp.clone()
    got4 = torch.full_like(q, 7.0)
    attention_bf16.decode_fused(got4, qkv, k4, v4, qw, kw, 1e-6, cos_sin, True, meta, meta.block_tables[0], page,
                                nq, nkv, D, 1 / math.sqrt(D), window, st, stream=False)
    assert torch.equal(k4, k2) and torch.equal(v4, v2)            # splits of a given length: the same cache
    assert torch.allclose(got4.float(), want.float(), rtol=2e-2, atol=2e-2)
    # reading another run's cache: nothing is written
    k3, v3 = k1.clone(), v1.clone()
    got3 = torch.zeros_like(q)
    ops().attention_decode_fused(got3, qkv, k3, v3, qw, kw, 1e-6, cos_sin, False, meta, meta.block_tables[0],
                                 page, nq, nkv, D, 1 / math.sqrt(D), window, st)
    assert torch.equal(k3, k1) and torch.equal(v3, v1)
    assert torch.allclose(got3.float(), want.float(), rtol=2e-2, atol=2e-2)


@pytest.mark.parametrize("window", [0, 100])
@pytest.mark.parametrize("ctas", [1, 2, 3, 5, 8])
@pytest.mark.parametrize("shape", [dict(D=128, nq=8, nkv=2, page=16), dict(D=64, nq=6, nkv=3, page=8), dict(D=128, nq=16, nkv=1, page=32),
                                   dict(D=64, nq=5, nkv=5, page=16)])
def test_decode_attention_in_a_cluster(shape, ctas, window):
    """A pair's splits as a cluster that finishes the pair: the bits and the cache of the same splits merged by a launch of
    its own.  Tokens of one split and of all, splits wholly behind a window, more splits asked for than the cluster has."""
    import ctypes
    from kipp_b200.csrc.build import load_library
    lib = load_library("attention_mma")
    p, i, ll, f = ctypes.c_void_p, ctypes.c_int, ctypes.c_longlong, ctypes.c_float
    head = [p, p, ll, p, p, p, p, i, f, p, i, p, p, p, i, i, p, i, i, i, i, f, i, i, p, i]
    lib.kipp_attn_decode_mma_fused.argtypes = head + [i, p, p, p]
    lib.kipp_attn_decode_cluster_fused.argtypes = head + [p, p]
    D, nq, nkv, page = shape["D"], shape["nq"], shape["nkv"], shape["page"]
    layout = [(700, 1), (15, 1), (63, 1), (64, 1), (1023, 1), (0, 1), (300, 1)]
    meta, table, _, kp, vp = attention_case(78, D, nq, nkv, page, layout, torch.bfloat16)
    T = meta.tokens
    g = torch.Generator().manual_seed(6)
    qkv = torch.randn(T, (nq + 2 * nkv) * D, generator=g).to(torch.bfloat16).to(DEV)
    qw, kw = ((1 + 0.2 * torch.randn(D, generator=g)).to(DEV) for _ in range(2))
    inv = torch.pow(torch.tensor(1e4, dtype=torch.float64), -(torch.arange(D // 2) * 2.0 / D).double()).float().to(DEV)
    cos_sin = ops().rope_table(meta.positions, inv, T)
    rows = torch.arange(T, dtype=torch.int32, device=DEV)
    tables = meta.block_tables[0]
    scratch = torch.full((T * nq * (ctas * (D + 2) + 1),), float("nan"), device=DEV)
    for keys in (64, 128):
        split_keys = torch.full((T,), keys, dtype=torch.int32, device=DEV)
        results = []
        for cluster in (False, True):
            k, v, st = kp.clone(), vp.clone(), status()
            out = torch.full((T, nq, D), 7.0, dtype=torch.bfloat16, device=DEV)
            args = [out.data_ptr(), qkv.data_ptr(), qkv.stride(0), k.data_ptr(), v.data_ptr(), qw.data_ptr(), kw.data_ptr(), 0, 1e-6,
                    cos_sin.data_ptr(), 1, meta.q_start.data_ptr(), meta.context_len.data_ptr(), tables.data_ptr(), tables.shape[1], page,
                    rows.data_ptr(), T, nq, nkv, D, 1 / math.sqrt(D), window, ctas, split_keys.data_ptr(), 1]
            stream = torch.cuda.current_stream().cuda_stream
            if cluster:
                rc = lib.kipp_attn_decode_cluster_fused(*args, st.data_ptr(), stream)
            else:
                rc = lib.kipp_attn_decode_mma_fused(*args, 0, scratch.data_ptr(), st.data_ptr(), stream)
            assert rc == 0 and st.tolist() == [0, 0, 0, 0]
            results.append((out, k, v))
        assert all(torch.equal(a, b) for a, b in zip(*results)), keys
        assert torch.isfinite(results[1][0].float()).all()


@pytest.mark.parametrize("window", [None, 500])
@pytest.mark.parametrize("shape", [dict(D=128, nq=8, nkv=2, page=16), dict(D=64, nq=6, nkv=3, page=32),
                                   dict(D=128, nq=16, nkv=1, page=16)])
def test_decode_attention_dealt_out_as_a_stream(shape, window):
    """Many decoded tokens of very different lengths: the key tiles of all (token, kv head)
    pairs are dealt out in equal runs to one wave of CTAs, so runs end inside pairs and span
    several short ones; every token against the plain reference, and against the kernel
    that cuts each token into splits of its own.  A far key that stands out must be found
    wherever the cuts fall."""
    from kipp_b200.kernels import attention_bf16
    D, nq, nkv, page = shape["D"], shape["nq"], shape["nkv"], shape["page"]
    rng = random.Random(D + nq)
    layout = [(rng.choice([0, 1, 63, 64, 65, 200, 1000, 2500, 4000]) + rng.randrange(3), 1) for _ in range(70)]
    layout[5] = (6000, 1)
    meta, table, q, kp, vp = attention_case(31, D, nq, nkv, page, layout, torch.bfloat16)
    # one key far back in the longest request that the query of that token points at
    e, far = 5, 777
    pg, slot = int(table[e, far // page]), far % page
    kp[pg, :, slot, :] = 0
    kp[pg, :, slot, 0] = 30.0
    q[e, :, :] = 0
    q[e, :, 0] = 30.0
    st = status()
    attention_bf16.decode_scratch(torch.device(DEV), meta.tokens, nq, D).fill_(float("nan"))
    out = torch.full_like(q, 9.0)
    attention_bf16.run("mma", out, q, kp, vp, meta, meta.block_tables[0], page, nq, nkv, D, 1 / math.sqrt(D), window, st)
    ref = attention_ref(meta, table, q, kp, vp, layout, page, window, 1 / math.sqrt(D))
    assert torch.allclose(out.double().cpu(), ref, rtol=2e-2, atol=2e-2)
    if window is None:                           # the far key takes all the weight
        assert torch.allclose(out[e].float().cpu(), vp[pg, :, slot, :].float().cpu().repeat_interleave(nq // nkv, 0),
                              rtol=2e-2, atol=2e-2)
    out1 = torch.full_like(q, 9.0)
    attention_bf16.run("mma", out1, q, kp, vp, meta, meta.block_tables[0], page, nq, nkv, D, 1 / math.sqrt(D), window,
                       st, stream=False)
    assert torch.allclose(out1.float(), out.float(), rtol=2e-2, atol=2e-2)
    assert st.tolist() == [0, 0, 0, 0]


@pytest.mark.parametrize("context,D", [(63, 128), (64, 64), (1022, 128), (1030, 64), (4094, 128)])
def test_decode_merge_at_its_edges(context, D):
    """One decoded token whose keys are cut into 1, 2, 16, 17 and 64 splits of a tile each: the merge fetches 16 splits
    at a time, in heads of half a warp and of a whole one.  What lies in the scratch beforehand must not matter."""
    from kipp_b200.kernels import attention_bf16
    nq, nkv, page, layout = 8, 2, 16, [(context, 1)]
    meta, table, q, kp, vp = attention_case(context, D, nq, nkv, page, layout, torch.bfloat16)
    out, st = torch.full_like(q, 9.0), status()
    attention_bf16.decode_scratch(torch.device(DEV), 1, nq, D).fill_(float("nan"))
    attention_bf16.run("mma", out, q, kp, vp, meta, meta.block_tables[0], page, nq, nkv, D, 1 / math.sqrt(D), None, st, stream=False)
    ref = attention_ref(meta, table, q, kp, vp, layout, page, None, 1 / math.sqrt(D))
    assert st.tolist() == [0, 0, 0, 0] and torch.allclose(out.double().cpu(), ref, rtol=2e-2, atol=2e-2)


def test_a_bounded_wait_runs_out_and_reports():
    """The give-up branch of the mbarrier wait every tensor-core kernel uses
    (csrc/mbarrier.cuh), run by a probe kernel on a barrier nothing arrives at, with
    a limit of some ten microseconds: the kernel returns by itself, the status word
    the engine reads is set, and the wait lasted as long as its limit."""
    import ctypes
    from kipp_b200.csrc.build import load_library
    lib = load_library("wait_probe")
    lib.kipp_wait_probe.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_longlong, ctypes.c_void_p]
    lib.kipp_wait_probe.restype = ctypes.c_int
    st = status()
    waited = torch.zeros(1, dtype=torch.int64, device=DEV)
    limit = 20_000
    rc = lib.kipp_wait_probe(st.data_ptr(), waited.data_ptr(), limit, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    assert rc == 0
    assert st.tolist() == [0, 1, 0, 0]
    assert limit <= int(waited) < 200 * limit


@pytest.mark.parametrize("late,limit,gives_up", [(0, 10_000_000, 0), (400_000, 10_000_000, 0), (9_000_000, 20_000, 1), (9_000_000, 0, 1)])
def test_a_cluster_outlives_what_is_sent_late(late, limit, gives_up):
    """A CTA whose wait for a neighbour's values ran out stays until the neighbour has sent them and they have landed
    (csrc/mbarrier.cuh: the end of the split products' and the decode attention's clusters): the status word is set, the
    word that came late lies in the mailbox, and the kernel returns by itself.  (A wait looks at its limit every 64 polls, which
    block for a while each: the late word comes some 5 ms after the others.)"""
    import ctypes
    from kipp_b200.csrc.build import load_library
    fn = load_library("wait_probe").kipp_mail_probe
    fn.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_longlong, ctypes.c_longlong, ctypes.c_int, ctypes.c_void_p]
    st, landed = status(), torch.zeros(1, dtype=torch.int32, device=DEV)
    for word in (77, 78, 79):
        assert fn(st.data_ptr(), landed.data_ptr(), late, limit, word, torch.cuda.current_stream().cuda_stream) == 0
        torch.cuda.synchronize()
        assert landed.item() == word
    assert st.tolist() == [0, gives_up, 0, 0]


@pytest.mark.parametrize("interleaved", [0, 1])
@pytest.mark.parametrize("D,rot_off,rot", [(64, 0, 64), (192, 128, 64), (192, 0, 16), (40, 8, 32), (72, 8, 24), (192, 128, 6), (48, 4, 40),
                                           (320, 24, 256)])
@pytest.mark.parametrize("dtype", DTYPES)
def test_head_segments_rotated(dtype, D, rot_off, rot, interleaved):
    """A rotated segment with a norm, in whole vectors where its rotated dims are that and an element at a time
    elsewhere (rotated parts that start or end inside a vector, rows or a rotation table off a 16-byte boundary), against
    float64: the value is rounded once to the result's type, and float32 on its way (a sum of D squares, three
    products and a sum)."""
    import ctypes
    from kipp_b200.csrc.build import load_library

    class Segment(ctypes.Structure):
        _fields_ = ([(n, ctypes.c_int) for n in ("src_off", "heads", "dim", "src_stride", "rot_off", "rot", "target", "dst_off", "dst_stride",
                                                 "heads_per_row", "norm_all", "interleaved", "unit_norm")]
                    + [(n, ctypes.c_void_p) for n in ("bias", "norm_w", "cos_sin", "dst")] + [("ld_dst", ctypes.c_longlong)])

    fn = load_library("head_ops").kipp_head_segments
    p, i, ll = ctypes.c_void_p, ctypes.c_int, ctypes.c_longlong
    fn.argtypes = [p, ll, i, p, i, p, p, i, i, i, p, p, p, i, i, i, i, ctypes.c_float, p, p]
    T, H, eps = 5, 3, 1e-6
    g = torch.Generator().manual_seed(D + rot)
    x = torch.randn(T, H, D, generator=g).to(dtype)
    w = torch.randn(D, generator=g)
    angle = torch.rand(T, rot // 2, generator=g) * 6
    cs = torch.stack([angle.cos(), angle.sin()], -1).contiguous()
    v = x.double()
    v = v / (v.square().mean(-1, keepdim=True) + eps).sqrt() * w.double()
    c, s = cs.double()[:, None, :, 0], cs.double()[:, None, :, 1]
    r = v[..., rot_off:rot_off + rot].clone()
    lo, hi = (r[..., 0::2], r[..., 1::2]) if interleaved else (r[..., :rot // 2], r[..., rot // 2:])
    turned = (lo * c - hi * s, hi * c + lo * s)
    v[..., rot_off:rot_off + rot] = torch.stack(turned, -1).flatten(-2) if interleaved else torch.cat(turned, -1)
    ulp = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -23
    bound = ulp * v.abs() + (D + 8) * 2.0 ** -24 * v.abs().amax()
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    bits = []
    for src_shift, w_shift, cs_shift in ((0, 0, 0), (0, 1, 0), (0, 0, 2), (1, 0, 0)):
        held = torch.zeros(src_shift + x.numel(), dtype=dtype, device=DEV)
        held[src_shift:] = x.flatten()
        norm, table = torch.zeros(w_shift + D, device=DEV), torch.zeros(cs_shift + cs.numel(), device=DEV)
        norm[w_shift:], table[cs_shift:] = w, cs.flatten()
        out = torch.zeros(T, H, D, dtype=dtype, device=DEV)
        seg = Segment(src_off=0, heads=H, dim=D, src_stride=D, rot_off=rot_off, rot=rot, target=0, dst_stride=D, interleaved=interleaved,
                      norm_w=norm[w_shift:].data_ptr(), cos_sin=table[cs_shift:].data_ptr(), dst=out.data_ptr(), ld_dst=H * D)
        rc = fn(held[src_shift:].data_ptr(), H * D, 0 if dtype == torch.float32 else 1, ctypes.byref(seg), 1, None, None, 0, 0, 0, None, None,
                None, 0, 1, T, 0, eps, status.data_ptr(), torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        assert rc == 0 and status.item() == 0
        assert ((out.double().cpu() - v).abs() <= bound).all(), (src_shift, w_shift, cs_shift)
        bits += [out] if src_shift == 0 else []                                  # (rows off 16 bytes add their squares otherwise)
    assert all(torch.equal(b, bits[0]) for b in bits)                            # whichever form turned them


@pytest.mark.parametrize("page", [8, 16, 64, 192, 24])
@pytest.mark.parametrize("sizes", [(72, 40, 8, 24, 3), (512, 128, 64, 128, 5), (40, 16, 0, 16, 2), (200, 64, 16, 256, 2)])
def test_latent_expand(sizes, page):
    """The heads' keys and values out of cached latents, on tcgen05 where the page sizes allow it and on mma.sync at any:
    entries of 1 token, of a page of the result less, exactly and plus one, and of several tiles, in pages of the pool that follow no
    order; ranks and features that end inside a step or tile.  Every value is a sum of `rank` products, in float32 (error
    under rank 2^-23 sum |c||w|), rounded once; the shared part is copied, rows past an entry's last token are zeros, and the
    rest of the result's pages stays untouched."""
    import ctypes
    from kipp_b200.csrc.build import load_library
    rank, dim, rot, v_dim, heads = sizes
    lens = [1, 63, 64, 65, 300]
    g = torch.Generator().manual_seed(rank + page)
    per = -(-max(lens) // page)
    n_pages = per * len(lens) + 3
    pool = torch.randn(n_pages, page, rank + rot, generator=g).bfloat16()
    order = torch.randperm(n_pages, generator=g)
    table = torch.full((len(lens), per), -1, dtype=torch.int32)
    at = 0
    for e, n in enumerate(lens):
        need = -(-n // page)
        table[e, :need] = order[at:at + need].int()
        at += need
    wk = (torch.randn(heads * dim, rank, generator=g) * 0.1).bfloat16()
    wv = (torch.randn(heads * v_dim, rank, generator=g) * 0.1).bfloat16()
    new = torch.tensor([1, 10, 64, 1, 299])                                   # tokens of the step, the others are cached before
    q_start = torch.cat([torch.zeros(1, dtype=torch.int64), new.cumsum(0)]).int().to(DEV)
    context = (torch.tensor(lens) - new).int().to(DEV)
    width = -(-per * page // 64)
    p, i = ctypes.c_void_p, ctypes.c_int
    rest = [p, i, i, i, p, p, i, p, p, i, i, i, i, i, p, p, p, i, p, p]
    dev = [x.to(DEV).contiguous() for x in (pool, table, wk, wv)]
    on_tc = load_library("attention_tc").kipp_attn_prefill_tc_page_ok(page)
    assert bool(on_tc) == (page != 24)
    bits = []
    for tc in ([True, False] if on_tc else [False]):
        fn = load_library("attention_tc").kipp_latent_expand_tc if tc else load_library("head_ops").kipp_latent_expand
        fn.argtypes = [p] + ([i] if tc else []) + rest
        ko = torch.full((len(lens), width, heads, 64, dim + rot), 7.0, dtype=torch.bfloat16, device=DEV)
        vo = torch.full((len(lens), width, heads, 64, v_dim), 7.0, dtype=torch.bfloat16, device=DEV)
        to = torch.zeros(len(lens), width, dtype=torch.int32, device=DEV)
        status = torch.zeros(8, dtype=torch.int32, device=DEV)
        rc = fn(dev[0].data_ptr(), *([n_pages] if tc else []), dev[1].data_ptr(), per, page, rank + rot, q_start.data_ptr(),
                context.data_ptr(), len(lens), dev[2].data_ptr(), dev[3].data_ptr(), rank, dim, rot, v_dim, heads, ko.data_ptr(),
                vo.data_ptr(), to.data_ptr(), width, status.data_ptr(), torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        assert rc == 0 and status.abs().sum().item() == 0
        assert torch.equal(to.cpu().flatten(), torch.arange(len(lens) * width, dtype=torch.int32))
        bits.append((ko, vo))
        for e, n in enumerate(lens):
            rows = torch.cat([pool[table[e, j]] for j in range(-(-n // page))])[:n]
            c = rows[:, :rank].double()
            end = -(-n // 64) * 64
            for out, w, size in ((ko, wk, dim), (vo, wv, v_dim)):
                got = out[e].cpu().double().transpose(1, 2).reshape(width * 64, heads, -1)
                ref = (c @ w.double().t()).reshape(n, heads, size)
                slack = (rank * 2.0 ** -23 * (c.abs() @ w.double().abs().t())).reshape(n, heads, size)
                assert ((got[:n, :, :size] - ref).abs() <= 2.0 ** -8 * ref.abs() + slack).all(), (tc, e)
                if out is ko:
                    assert (got[:n, :, size:] == rows[:, None, rank:].double()).all(), (tc, e)
                assert (got[n:end] == 0).all() and (got[end:] == 7).all(), (tc, e)
    assert all(torch.equal(b[k], bits[0][k]) for b in bits for k in (0, 1))          # the engine takes either by their sizes


@pytest.mark.parametrize("window", [0, 40])
@pytest.mark.parametrize("sizes", [(20, 96, 64), (16, 576, 512), (33, 1312, 24)])
def test_attention_shared_key(sizes, window):
    """One key row per token for all heads, its head the value: tokens at the edges of the tiles of 32 keys, in pages of any
    order, as few blocks (two stages of keys where they fit; 1,312 columns leave room for one), as many (one stage) and cut
    into runs.  Without runs a token has the same bits among few and among many; all stay within the bound of 16-bit inputs
    and results (weights as pairs of bfloat16, sums in float32) around float64."""
    import ctypes
    from kipp_b200.csrc.build import load_library
    n_q, D, V = sizes
    page, width, scale = 16, 14, 0.05
    g = torch.Generator().manual_seed(D + window)
    at = [0, 1, 30, 31, 32, 63, 64, 95, 96, 200]
    T = 300
    pos = torch.tensor((at * T)[:T], dtype=torch.int32)
    entry = torch.arange(T, dtype=torch.int32) % 3
    table = torch.randperm(3 * width, generator=g).int().reshape(3, width)
    pool = torch.randn(3 * width, page, D, generator=g).bfloat16()
    q = torch.randn(T, n_q, D, generator=g).bfloat16()
    fn = load_library("attention_mix").kipp_attention_shared_key
    p, i, f = ctypes.c_void_p, ctypes.c_int, ctypes.c_float
    fn.argtypes = [p, p, p, p, p, p, i, i, i, i, i, i, f, i, f, i, p, p, p, p]
    d = [x.to(DEV) for x in (q, pool, pos, entry, table)]
    status = torch.zeros(8, dtype=torch.int32, device=DEV)

    def run(tokens, runs):
        out = torch.zeros(tokens, n_q, V, dtype=torch.bfloat16, device=DEV)
        partial = torch.zeros(tokens * runs * n_q * (V + 2), device=DEV)
        rc = fn(out.data_ptr(), d[0].data_ptr(), d[1].data_ptr(), d[2].data_ptr(), d[3].data_ptr(), d[4].data_ptr(), width, page, tokens,
                n_q, D, V, scale, window, 1.0, runs, partial.data_ptr(), None, status.data_ptr(), torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        assert rc == 0 and status.abs().sum().item() == 0
        return out

    many, few, cut = run(T, 1), run(len(at), 1), run(len(at), 4)
    assert torch.equal(many[:len(at)], few)
    for t in range(len(at)):
        lo = max(0, int(pos[t]) - window + 1) if window else 0
        keys = torch.cat([pool[j] for j in table[int(entry[t])]])[lo:int(pos[t]) + 1].double()
        w = torch.softmax(q[t].double() @ keys.t() * scale, -1)
        want, size = w @ keys[:, :V], w @ keys[:, :V].abs()
        for got in (few[t], cut[t]):
            assert ((got.double().cpu() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-4 * size).all(), (t, window)


@pytest.mark.parametrize("lens", [[37], [1, 1, 1]])
@pytest.mark.parametrize("heads,v_dim,norm_groups", [(8, 64, 1), (8, 64, 8), (64, 64, 1), (192, 64, 1), (5, 36, 1), (6, 20, 3)])
def test_gated_norm_adds_in_one_order(heads, v_dim, norm_groups, lens):
    """The gate and grouped norm behind the state space scan take four channels at a time where the gate's rows start on
    that, one channel elsewhere and in parts too long for shared memory: the same bits in 32-bit, for prompts and one-token
    steps, in parts of fewer and of more channels than threads."""
    import ctypes
    from kipp_b200.csrc.build import load_library
    lib = load_library("recurrent")
    p, i, ll, f = ctypes.c_void_p, ctypes.c_int, ctypes.c_longlong, ctypes.c_float
    lib.kipp_ssd_scan.argtypes = [p, ll, p, ll, i, i, i, i, p, p, i, p, p, p, p, i, p, ll, p, p, p, i, i, i, i, i, i, f, p, p, p]
    lib.kipp_ssd_state_floats.restype = lib.kipp_recurrent_scratch_floats.restype = ll
    D, taps, T, E = 16, 3, sum(lens), len(lens)
    inner, channels = heads * v_dim, heads * v_dim + 2 * D
    g = torch.Generator().manual_seed(heads + v_dim)
    rnd = lambda *s: torch.randn(*s, generator=g).to(DEV)                      # noqa: E731
    x, z, dt = rnd(T, channels), rnd(T, inner), rnd(T, heads)
    weights = [rnd(taps, channels) * 0.5, rnd(channels) * 0.1, rnd(heads), rnd(heads) * 0.5, rnd(heads), rnd(inner)]
    stride = lib.kipp_ssd_state_floats(heads, 1, D, v_dim, taps)
    state = rnd(E, stride)
    q_start = torch.tensor([0] + np.cumsum(lens).tolist(), dtype=torch.int32, device=DEV)
    entry = torch.repeat_interleave(torch.arange(E), torch.tensor(lens)).int().to(DEV)
    slots = torch.arange(E, dtype=torch.int32, device=DEV)
    results = []
    for shift in (0, 1):
        ld = channels + heads + (-heads) % 4 + inner + 4
        z_off = ld - inner - 4 + shift
        proj = torch.zeros(T, ld, device=DEV)
        proj[:, :channels], proj[:, channels:channels + heads], proj[:, z_off:z_off + inner] = x, dt, z
        out, s = torch.zeros(T, inner, device=DEV), state.clone()
        scratch = torch.zeros(lib.kipp_recurrent_scratch_floats(T, heads, D, v_dim, 4), device=DEV)
        conv = torch.zeros(T, channels, device=DEV)
        w = [t.data_ptr() for t in weights]
        rc = lib.kipp_ssd_scan(out.data_ptr(), inner, proj.data_ptr(), ld, 0, z_off, 0, channels, w[0], w[1], taps, w[2], w[3], w[4], w[5],
                               norm_groups, s.data_ptr(), stride, q_start.data_ptr(), entry.data_ptr(), slots.data_ptr(), E, T, heads, 1, D,
                               v_dim, 1e-5, scratch.data_ptr(), conv.data_ptr(), torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        assert rc == 0 and torch.isfinite(out).all()
        results.append((out, s))
    assert torch.equal(results[0][0], results[1][0]) and torch.equal(results[0][1], results[1][1])


@pytest.mark.parametrize("D,v_dim,heads,n", [(128, 64, 4, 53), (32, 36, 3, 16), (64, 32, 2, 18), (100, 64, 2, 5), (256, 20, 2, 35), (16, 64, 1, 6)])
def test_state_space_scans_add_in_one_order(D, v_dim, heads, n):
    """The scan has a leaf of rows a thread where there are few blocks and two where they crowd the SMs: an entry's outputs and
    its state have the same bits alone and among as many as that takes, for whole groups of four tokens and rests, heads
    of whole leaves and others, columns that end inside a block's."""
    import ctypes
    from kipp_b200.csrc.build import load_library
    lib = load_library("recurrent")
    p, i, ll, f = ctypes.c_void_p, ctypes.c_int, ctypes.c_longlong, ctypes.c_float
    lib.kipp_ssd_scan.argtypes = [p, ll, p, ll, i, i, i, i, p, p, i, p, p, p, p, i, p, ll, p, p, p, i, i, i, i, i, i, f, p, p, p]
    lib.kipp_ssd_state_floats.restype = lib.kipp_recurrent_scratch_floats.restype = ll
    taps, inner = 2, heads * v_dim
    channels, sms = inner + 2 * D, torch.cuda.get_device_properties(0).multi_processor_count
    stride = lib.kipp_ssd_state_floats(heads, 1, D, v_dim, taps)
    g = torch.Generator().manual_seed(D + n)
    rnd = lambda *s: torch.randn(*s, generator=g).to(DEV)                      # noqa: E731
    z_off, ld = channels + heads + (-heads) % 4, channels + heads + (-heads) % 4 + inner
    rows, first = rnd(n, ld), rnd(1, stride)
    weights = [rnd(taps, channels) * 0.5, rnd(channels) * 0.1, rnd(heads), rnd(heads) * 0.5, rnd(heads), rnd(inner)]
    w = [t.data_ptr() for t in weights]

    def run(E):
        T = E * n
        proj, state = rows.repeat(E, 1).contiguous(), first.repeat(E, 1).contiguous()
        q_start = torch.arange(0, T + 1, n, dtype=torch.int32, device=DEV)
        entry, slots = torch.arange(E, device=DEV).repeat_interleave(n).int(), torch.arange(E, dtype=torch.int32, device=DEV)
        out, conv = torch.zeros(T, inner, device=DEV), torch.zeros(T, channels, device=DEV)
        scratch = torch.zeros(lib.kipp_recurrent_scratch_floats(T, heads, D, v_dim, 4), device=DEV)
        rc = lib.kipp_ssd_scan(out.data_ptr(), inner, proj.data_ptr(), ld, 0, z_off, 0, channels, w[0], w[1], taps, w[2], w[3], w[4], w[5],
                               1, state.data_ptr(), stride, q_start.data_ptr(), entry.data_ptr(), slots.data_ptr(), E, T, heads, 1, D,
                               v_dim, 1e-5, scratch.data_ptr(), conv.data_ptr(), torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        assert rc == 0 and torch.isfinite(out).all()
        return out.reshape(E, n, inner), state
    (one, kept), E = run(2), 4 * sms // heads + 1
    many, states = run(E)
    assert torch.equal(many, one[:1].expand_as(many)) and torch.equal(states, kept[:1].expand_as(states))


@pytest.mark.parametrize("D,v_dim,heads,lens", [(128, 64, 20, [53, 1, 7]), (64, 36, 64, [16, 40]), (100, 64, 30, [21]), (256, 32, 40, [9, 30]),
                                                (32, 32, 130, [6, 33, 1])])
def test_state_space_scans_of_either_form(D, v_dim, heads, lens):
    """A leaf of rows a thread and two, as the longest entry's length chooses: the same bits."""
    import ctypes
    from kipp_b200.csrc.build import load_library
    lib = load_library("recurrent")
    p, i, ll, f = ctypes.c_void_p, ctypes.c_int, ctypes.c_longlong, ctypes.c_float
    lib.kipp_ssd_scan_of.argtypes = [p, ll, p, ll, i, i, i, i, p, p, i, p, p, p, p, i, p, ll, p, p, p, i, i, i, i, i, i, i, f, p, p, p]
    lib.kipp_ssd_state_floats.restype = lib.kipp_recurrent_scratch_floats.restype = ll
    taps, inner, E, T = 2, heads * v_dim, len(lens), sum(lens)
    channels = inner + 2 * D
    stride = lib.kipp_ssd_state_floats(heads, 1, D, v_dim, taps)
    g = torch.Generator().manual_seed(D)
    rnd = lambda *s: torch.randn(*s, generator=g).to(DEV)                      # noqa: E731
    z_off = channels + heads + (-heads) % 4
    ld = z_off + inner
    proj, first = rnd(T, ld), rnd(E, stride)
    weights = [rnd(taps, channels) * 0.5, rnd(channels) * 0.1, rnd(heads), rnd(heads) * 0.5, rnd(heads), rnd(inner)]
    w = [t.data_ptr() for t in weights]
    q_start = torch.tensor([0] + lens).cumsum(0).int().to(DEV)
    entry, slots = torch.arange(E).repeat_interleave(torch.tensor(lens)).int().to(DEV), torch.arange(E, dtype=torch.int32, device=DEV)
    results = []
    for longest, leaves in ((T, 1), (1, 2)):
        assert lib.kipp_ssd_scan_leaves(D, v_dim, heads, E, T, longest) == leaves
        state, out, conv = first.clone(), torch.zeros(T, inner, device=DEV), torch.zeros(T, channels, device=DEV)
        scratch = torch.zeros(lib.kipp_recurrent_scratch_floats(T, heads, D, v_dim, 4), device=DEV)
        rc = lib.kipp_ssd_scan_of(out.data_ptr(), inner, proj.data_ptr(), ld, 0, z_off, 0, channels, w[0], w[1], taps, w[2], w[3], w[4], w[5],
                                  1, state.data_ptr(), stride, q_start.data_ptr(), entry.data_ptr(), slots.data_ptr(), E, T, longest, heads, 1,
                                  D, v_dim, 1e-5, scratch.data_ptr(), conv.data_ptr(), torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        assert rc == 0 and torch.isfinite(out).all()
        results.append((out, state))
    assert all(torch.equal(a, b) for a, b in zip(*results))


@pytest.mark.parametrize("size", [1, 100, 128, 2048, 2049, 2560, 5000])
@pytest.mark.parametrize("dtype", DTYPES)
def test_row_dot(dtype, size):
    """A weight's product with each row: thread t of 128 adds elements t, t + 128, ... in turn, then the threads' sums meet
    lane by lane, the farthest first, and warp by warp: that order's bits, whatever the alignment."""
    import ctypes
    from kipp_b200.csrc.build import load_library
    fn = load_library("elementwise").kipp_row_dot
    p, i, ll = ctypes.c_void_p, ctypes.c_int, ctypes.c_longlong
    fn.argtypes = [p, p, ll, i, p, i, i, p]
    rows = 3
    g = torch.Generator().manual_seed(size)
    # 8-bit mantissas: products are exact in 32 bits, so an FMA is a rounded addition
    x, w = torch.randn(rows, size, generator=g).bfloat16().float(), torch.randn(size, generator=g).bfloat16().float()
    prod = torch.zeros(rows, -(-size // 128) * 128)
    prod[:, :size] = x * w
    acc = torch.zeros(rows, 128)
    for part in prod.reshape(rows, -1, 128).unbind(1):
        acc = acc + part

    def lanes(v):                                                                # [..., 32]: the butterfly of a warp
        for o in (16, 8, 4, 2, 1):
            v = v[..., :o] + v[..., o:2 * o]
        return v[..., 0]

    warps = torch.zeros(rows, 32)
    warps[:, :4] = lanes(acc.reshape(rows, 4, 32))
    want = lanes(warps)
    for shift in (0, 1):
        held = torch.zeros(rows, size + 3, dtype=dtype, device=DEV)
        held[:, shift:shift + size] = x
        wd, out = torch.zeros(size + 1, device=DEV), torch.zeros(rows, device=DEV)
        wd[shift:shift + size] = w
        rc = fn(out.data_ptr(), held[:, shift:].data_ptr(), size + 3, 0 if dtype == torch.float32 else 1, wd[shift:].data_ptr(), rows, size,
                torch.cuda.current_stream().cuda_stream)
        assert rc == 0 and torch.equal(out.cpu(), want)


@pytest.mark.parametrize("vocab", [51, 700, 40001])
def test_sample_rows_below_an_infinite_value(vocab):
    """Under a largest value that is not finite every candidate weighs e^(inf - inf).  Such a total counts 2^63 units a
    candidate modulo 2^64, so of an odd number of candidates the last is drawn and of an even number the first (the last
    without a nucleus); the sums of a NaN's weight in a draw are none."""
    from kipp_b200.kernels import sampling as ks
    x = torch.randn(6, vocab, generator=torch.Generator().manual_seed(vocab)) * 2
    x[0, 7] = x[1, 7] = x[1, 9] = x[2, 7] = x[2, 9] = x[2, 40] = math.inf
    x[3] = -math.inf
    x[4] = 3e38                                                                  # infinite once divided by the temperature
    x[5, ::2] = math.nan
    x[5, 1] = math.inf
    first = {0: 7, 1: 7, 2: 7, 3: 0, 4: 0, 5: 1}
    last = {0: 7, 1: 9, 2: 40, 3: vocab - 1, 4: vocab - 1, 5: 1}
    odd = {0: True, 1: False, 2: True, 3: vocab % 2 == 1, 4: vocab % 2 == 1, 5: True}
    t = lambda v, d: torch.full((6,), v, dtype=d, device=DEV)                     # noqa: E731
    for top_p, min_p in ((0.9, 0.0), (0.3, 0.5), (1.0, 0.0)):
        for u in (0.0, 0.4, 0.999):
            got = ks.sample_rows(x.to(DEV), t(1e-3, torch.float32), t(0, torch.int32), t(top_p, torch.float32), t(min_p, torch.float32),
                                 t(u, torch.float64)).tolist()
            assert got == [last[r] if odd[r] or top_p == 1.0 else first[r] for r in range(6)], (top_p, u)
    got = ks.sample_rows(x.to(DEV), t(1e-3, torch.float32), t(5, torch.int32), t(0.9, torch.float32), t(0.0, torch.float32), t(0.4, torch.float64))
    assert got.tolist()[3:5] == [4, 4]                                           # five candidates are left


@pytest.mark.parametrize("entries,longest", [(1, 0), (400, 0), (400, 2), (400, 800)])
@pytest.mark.parametrize("D,V", [(32, 32), (64, 20), (128, 64), (100, 36), (256, 32)])
def test_gated_delta_scans_add_in_one_order(D, V, entries, longest):
    """The output's sum over the key rows, with a thread per column (few warps at work, or said to
    be few by the longest entry's length) and four columns per thread (many): a thread's
    pairs of neighbouring rows by turns into two sums, those, then the lanes, the farthest first.  With equal queries, no
    decay and no write a column of the state that holds 2^30, 1 and -2^30 gives the query's value or 0, as the order
    meets the three; float32 sums of the state in that order say which."""
    import ctypes
    from kipp_b200.csrc.build import load_library
    lib = load_library("recurrent")
    p, i, ll, f = ctypes.c_void_p, ctypes.c_int, ctypes.c_longlong, ctypes.c_float
    lib.kipp_gated_delta_scan.argtypes = [p, ll, p, ll, i, i, i, p, i, p, ll, p, p, p, ll, i, p, p, ll, p, p, p, i, i, i, i, i, i, i, f, f, f, p, p, p]
    lib.kipp_recurrent_scratch_floats.restype = lib.kipp_gated_delta_state_floats.restype = ll
    heads, T = 2, 2 * entries
    blocks = entries * heads * -(-V // 8)
    assert blocks <= 64 or 2 * blocks > 148 * 12
    g = torch.Generator().manual_seed(D + V)
    state = torch.zeros(entries, heads, D, V)
    rows = torch.stack([torch.randperm(D, generator=g)[:3] for _ in range(entries * heads * V)]).reshape(entries, heads, V, 3)
    for n, value in enumerate((2.0 ** 30, 1.0, -2.0 ** 30)):
        state.scatter_(2, rows[..., n][:, :, None, :], value)
    P, R = (8, 4) if D <= 32 else (16, 4) if D <= 64 else (32, 4) if D <= 128 else (32, 8)
    padded = torch.zeros(entries, heads, P * R, V)
    padded[:, :, :D] = state
    by_lane = padded.reshape(entries, heads, R // 4, P, 2, 2, V)                  # row 4 (lane + P q) + 2 pair + half
    sums = [0.0, 0.0]
    for q in range(R // 4):
        for pair in range(2):
            sums[pair] = by_lane[:, :, q, :, pair] + sums[pair]                   # [.., lane, half, V]
    v = (sums[0][..., 0, :] + sums[0][..., 1, :]) + (sums[1][..., 0, :] + sums[1][..., 1, :])
    while v.shape[2] > 1:
        half = v.shape[2] // 2
        v = v[:, :, :half] + v[:, :, half:]
    want = v[:, :, 0]
    assert (want == 0).any() and (want == 1).any()
    channels = 2 * D + heads * V
    ld = channels + heads + (-channels - heads) % 4
    proj = torch.ones(T, ld, device=DEV)
    proj[:, channels:] = -200.0                                                   # write rates of 0
    ones = torch.ones(max(heads * D, channels, heads * V, V), device=DEV)
    a_raw, a_log = torch.full((T, heads * D), -300.0, device=DEV), torch.zeros(heads, device=DEV)      # decays of 1
    g_raw = torch.ones(T, heads * V, device=DEV)
    q_start = torch.arange(entries + 1, dtype=torch.int32, device=DEV) * 2
    entry = (torch.arange(T, device=DEV) // 2).int()
    slots = torch.arange(entries, dtype=torch.int32, device=DEV)
    S = state.reshape(entries, -1).to(DEV).clone()
    assert S.shape[1] == lib.kipp_gated_delta_state_floats(heads, 1, D, V, 1)
    scratch = torch.zeros(lib.kipp_recurrent_scratch_floats(T, heads, D, V, 5), device=DEV)
    conv, out = torch.zeros(T, channels, device=DEV), torch.zeros(T, heads, V, device=DEV)
    rc = lib.kipp_gated_delta_scan(out.data_ptr(), heads * V, proj.data_ptr(), ld, 0, 0, channels, ones.data_ptr(), 1, a_raw.data_ptr(),
                                   heads * D, ones.data_ptr(), a_log.data_ptr(), g_raw.data_ptr(), heads * V, 1, ones.data_ptr(), S.data_ptr(),
                                   S.shape[1], q_start.data_ptr(), entry.data_ptr(), slots.data_ptr(), entries, T, longest, heads, 1, D, V, 1.0, 1e-12,
                                   1.0, scratch.data_ptr(), conv.data_ptr(), torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    assert rc == 0 and torch.equal(S.cpu(), state.reshape(entries, -1))
    got = out.cpu().reshape(entries, 2, heads, V)
    for t in range(2):
        assert torch.equal(got[:, t] != 0, want != 0)


@pytest.mark.parametrize("hidden,outputs", [(512, 18), (1028, 64), (33, 5), (2560, 3)])
@pytest.mark.parametrize("dtype", DTYPES)
def test_routing_of_a_token_among_others(dtype, hidden, outputs):
    """A token's experts and weights have the same bits whether its block has an SM to itself with up to 32 warps (148 tokens), shares
    one with up to 16 (149, 255) or holds four tokens (256, 257), by logits and by scores, in rows of whole fours and others; the
    weights are the softmax of the chosen logits, whose sums of `hidden` products are float32."""
    import ctypes
    from kipp_b200.csrc.build import load_library
    lib = load_library("moe")
    p, i, ll, f = ctypes.c_void_p, ctypes.c_int, ctypes.c_longlong, ctypes.c_float
    lib.kipp_moe_route.argtypes = [p, p, p, ll, i, p, p, i, i, i, i, p]
    lib.kipp_moe_route_scores.argtypes = [p, p, p, ll, i, p, p, i, i, i, i, i, i, i, f, p]
    g = torch.Generator().manual_seed(hidden)
    h, w, b = torch.randn(257, hidden, generator=g).to(dtype).to(DEV), (torch.randn(outputs, hidden, generator=g) * 0.2).to(DEV), torch.randn(outputs, generator=g).to(DEV)
    top, code = min(3, outputs), 0 if dtype == torch.float32 else 1
    for scores in (False, True):
        kept = None
        for tokens in (257, 1, 33, 148, 149, 255, 256):
            expert, weight = torch.full((tokens, top), -9, dtype=torch.int32, device=DEV), torch.zeros(tokens, top, device=DEV)
            at = (expert.data_ptr(), weight.data_ptr(), h.data_ptr(), hidden, code, w.data_ptr(), b.data_ptr(), tokens, hidden, outputs)
            stream = torch.cuda.current_stream().cuda_stream
            rc = lib.kipp_moe_route_scores(*at, outputs, top, 1, 1, 1.5, stream) if scores else lib.kipp_moe_route(*at, top, stream)
            assert rc == 0
            kept = kept or (expert, weight)
            assert torch.equal(expert, kept[0][:tokens]) and torch.equal(weight, kept[1][:tokens]), (scores, tokens)
        if not scores:
            logits = (h.double() @ w.double().t() + b.double()).cpu()
            best = torch.gather(logits, 1, kept[0].long().cpu())
            slack = hidden * 2.0 ** -23 * float((h.double().abs() @ w.double().abs().t()).max()) + 1e-6
            assert (logits.topk(top).values - best <= 2 * slack).all()
            assert torch.allclose(kept[1].double().cpu(), torch.softmax(best, -1), atol=2 * slack)
