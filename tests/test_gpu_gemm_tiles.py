"""Plain tiles of 64, 128 and 256 columns with the factor per row, and ragged row tiles of the pair kernel."""
import pytest
import torch

from test_gpu_kernels import rel, rnd

pytestmark = pytest.mark.gpu
DEV = "cuda"


def scaled_case(M, N, K, chunks=3, eps=1e-6):
    x, w = rnd(M, K, dtype=torch.bfloat16, seed=31), rnd(N, K, dtype=torch.bfloat16, seed=32, scale=0.2)
    sumsq = rnd(M, chunks, seed=33).abs() + 0.1
    factor = torch.rsqrt(sumsq.double().sum(1) / K + eps)
    return x, w, sumsq, (x.double() @ w.double().T) * factor[:, None]


@pytest.mark.parametrize("M", [128, 129, 517, 1100])
@pytest.mark.parametrize("N,K", [(192, 128), (520, 200)])
@pytest.mark.parametrize("kernel", [64, 128, 256, "pair"])
@pytest.mark.parametrize("swiglu", [False, True])
def test_rows_without_their_factor(M, N, K, kernel, swiglu):
    from purhie_b200.csrc import gemm100
    x, w, sumsq, y = scaled_case(M, N, K)
    ref = torch.nn.functional.silu(y[:, 0::2]) * y[:, 1::2] if swiglu else y
    kw = dict(swiglu=swiglu, row_sumsq=sumsq, row_width=K, row_eps=1e-6)
    for dtype, bound in ((torch.float32, 2e-5), (torch.bfloat16, 5e-3)):     # sums in float32; a bfloat16 result is rounded once
        out = torch.full((M, N // 2 if swiglu else N), float("nan"), dtype=dtype, device=DEV)
        if kernel == "pair":
            gemm100.gemm_pair(x, w, out, **kw)
        else:
            gemm100.gemm(x, w, out, swapped=False, block_n=kernel, **kw)
        gemm100.check_errors(DEV)
        assert not torch.isnan(out).any()
        assert rel(out, ref) < bound


@pytest.mark.parametrize("M", [257, 300, 513, 640])
def test_pair_kernel_leaves_what_lies_behind_its_rows_alone(M):
    """Warps whose rows lie behind the last one skip their epilogue: float32, partial sums, bfloat16 and the addition."""
    from purhie_b200.csrc import gemm100
    N, K = 384, 256
    x, w = rnd(M, K, dtype=torch.bfloat16, seed=41), rnd(N, K, dtype=torch.bfloat16, seed=42)
    ref = x.double() @ w.double().T
    for dtype, splits, add in ((torch.float32, 1, False), (torch.float32, 2, False), (torch.bfloat16, 1, False), (torch.float32, 1, True)):
        size = splits * M * N
        held = torch.full((size + 512 * N,), 7.0, dtype=dtype, device=DEV)      # what lies behind out
        out = held[:size].view((splits, M, N) if splits > 1 else (M, N))
        gemm100.gemm_pair(x, w, out, splits=splits, accumulate=add)
        gemm100.check_errors(DEV)
        got = out.double().sum(0) if splits > 1 else out.double()
        assert rel(got, ref + 7.0 if add else ref) < (3e-5 if dtype == torch.float32 else 5e-3)
        assert (held[size:] == 7.0).all()


def guarded(shape, dtype, fill, behind=4096):
    """An array with `behind` sevens behind it in memory."""
    size = 1
    for d in shape:
        size *= d
    held = torch.full((size + behind,), 7.0, dtype=dtype, device=DEV)
    held[:size] = fill
    return held[:size].view(shape), held[size:]


@pytest.mark.parametrize("M,N,K", [(128, 192, 64), (130, 257, 200), (517, 518, 1032), (300, 1026, 4104)])
@pytest.mark.parametrize("block_n", [64, 128])
def test_narrow_tiles_add_into_the_output(M, N, K, block_n):
    """Out += product on tiles of 64 and 128 columns (rows of a multiple of 4 and not), with the bits of wide tiles."""
    from purhie_b200.csrc import gemm100
    x, w = rnd(M, K, dtype=torch.bfloat16, seed=51), rnd(N, K, dtype=torch.bfloat16, seed=52, scale=0.2)
    outs = []
    for bn in (block_n, 256):
        out, behind = guarded((M, N), torch.float32, 3.0)
        gemm100.gemm(x, w, out, swapped=False, block_n=bn, accumulate=True)
        gemm100.check_errors(DEV)
        assert (behind == 7.0).all()
        outs.append(out)
    assert torch.equal(outs[0], outs[1])
    assert rel(outs[0] - 3.0, x.double() @ w.double().T) < 3e-5


@pytest.mark.parametrize("M,N,K,splits", [(128, 192, 1024, 2), (300, 520, 3080, 3), (517, 1026, 8200, 8), (129, 130, 4096, 4)])
def test_k_in_parts_has_the_same_bits_on_all_tiles(M, N, K, splits):
    """K long enough for the ring of stages to wrap behind the weight tiles that were asked for early."""
    from purhie_b200.csrc import gemm100
    x, w = rnd(M, K, dtype=torch.bfloat16, seed=53), rnd(N, K, dtype=torch.bfloat16, seed=54, scale=0.2)
    outs = []
    for kernel in (64, 128, 256, "pair"):
        out, behind = guarded((splits, M, N), torch.float32, float("nan"))
        if kernel == "pair":
            gemm100.gemm_pair(x, w, out, splits=splits)
        else:
            gemm100.gemm(x, w, out, swapped=False, block_n=kernel, splits=splits)
        gemm100.check_errors(DEV)
        assert (behind == 7.0).all()
        outs.append(out)
    assert all(torch.equal(outs[0], o) for o in outs[1:])
    assert rel(outs[0].double().sum(0), x.double() @ w.double().T) < 3e-5


@pytest.mark.parametrize("M,N,K", [(128, 192, 64), (517, 520, 1032), (1100, 1024, 2048)])
@pytest.mark.parametrize("swiglu", [False, True])
def test_whole_sums_have_the_same_bits_on_all_tiles(M, N, K, swiglu):
    from purhie_b200.csrc import gemm100
    x, w, sumsq, _ = scaled_case(M, N, K)
    kw = dict(swiglu=swiglu, row_sumsq=sumsq, row_width=K, row_eps=1e-6)
    outs = []
    for kernel in (64, 128, 256, "pair"):
        out = torch.full((M, N // 2 if swiglu else N), float("nan"), dtype=torch.bfloat16, device=DEV)
        if kernel == "pair":
            gemm100.gemm_pair(x, w, out, **kw)
        else:
            gemm100.gemm(x, w, out, swapped=False, block_n=kernel, **kw)
        gemm100.check_errors(DEV)
        outs.append(out)
    assert all(torch.equal(outs[0], o) for o in outs[1:])


@pytest.mark.parametrize("M,N,K", [(128, 200, 64), (517, 1024, 520), (2048, 2304, 1024)])
@pytest.mark.parametrize("block_n", [64, 128, 256])
def test_a_weight_that_the_kernel_in_front_makes(M, N, K, block_n):
    """A plain product is complete when its w is the result of the kernel in front, which lets its dependents start early."""
    from purhie_b200.csrc import gemm100
    a, b, x = (rnd(r, c, dtype=torch.bfloat16, seed=s, scale=0.1) for r, c, s in ((N, 4096, 61), (K, 4096, 62), (M, K, 63)))
    w, out = torch.empty(N, K, dtype=torch.bfloat16, device=DEV), torch.empty(M, N, device=DEV)
    gemm100.gemm(a, b, w, swapped=False, block_n=256)
    torch.cuda.synchronize()
    ref = x.double() @ w.double().T
    for _ in range(4):
        w.fill_(float("nan"))
        out.fill_(float("nan"))
        gemm100.gemm(a, b, w, swapped=False, block_n=256)
        gemm100.gemm(x, w, out, swapped=False, block_n=block_n)
        gemm100.check_errors(DEV)
        assert rel(out, ref) < 3e-5
    early = torch.empty_like(out)
    gemm100.gemm(x, w, early, swapped=False, block_n=block_n, early_w=True)     # (w is complete by now)
    assert torch.equal(early, out)
