"""The float32 product and attention kernels give, bit for bit, what the plain kernels give: an operand that does not start
on 16 bytes goes to the plain kernel, whose additions run in the same order."""
import math

import pytest
import torch

from test_gpu_kernels import paged_case, rnd

pytestmark = pytest.mark.gpu
DEV = "cuda"


def off_by_one(x):
    """The same numbers one float32 behind a 16-byte boundary."""
    held = torch.empty(x.numel() + 4, device=DEV)
    y = held[1:1 + x.numel()].view(x.shape)
    y.copy_(x)
    assert y.data_ptr() % 16 == 4
    return y


# rows at and around the places where the kernel changes (1, 2, 4, 8, 16 | tiles); columns at and around 8, 32, 64, 128, the
# changes of the few-row plan (16 and 32 columns an SM) and a wide output; K around the chunks of 32 and 128
@pytest.mark.parametrize("M", [1, 2, 3, 4, 5, 8, 9, 16, 17, 33, 70, 129, 300])
@pytest.mark.parametrize("N,K", [(1, 4), (8, 96), (40, 124), (65, 132), (130, 224), (2376, 260), (4744, 128), (9001, 36)])
def test_float32_product_adds_in_the_plain_kernels_order(M, N, K):
    from purhie_b200.csrc import ops
    x, w = rnd(M, K, seed=M), rnd(N, K, seed=N)
    out, plain = torch.full((M, N), float("nan"), device=DEV), torch.full((M, N), float("nan"), device=DEV)
    ops.gemm_simple(x, w, out)
    ops.gemm_simple(off_by_one(x), w, plain)
    assert torch.equal(out, plain)
    # K products, each exact inside one rounded multiply-add: at most K half units in the last place of the sum of magnitudes
    bound = K * 2.0 ** -24 * (x.abs().double() @ w.abs().double().T)
    assert ((out.double() - x.double() @ w.double().T).abs() <= bound).all()


# K shared out among warps (three blocks of 128 and more): a round that is full, one that is not, a block of four numbers; columns up
# to the most that the few-row form takes; tiles in four groups, in two and in one
@pytest.mark.parametrize("M", [1, 2, 4, 7, 8, 16, 32, 139, 300])
@pytest.mark.parametrize("N,K", [(9, 260), (64, 1024), (1000, 3076), (2368, 388), (2368, 1028), (8200, 300)])
def test_float32_product_shares_k_out_in_the_plain_kernels_order(M, N, K):
    test_float32_product_adds_in_the_plain_kernels_order(M, N, K)


# decoded tokens alone (rows kernel), portions long enough for tiles beside decoded tokens, a portion of three tokens, portions
# that start mid-context; block edges of 32 and 128 keys; enough rows for tiles of eight rows a warp
CASES = [[(1, 1), (32, 1), (33, 1), (128, 1), (129, 1), (300, 1)],
         [(40, 40), (1, 1), (129, 1), (161, 33), (300, 3), (260, 5), (64, 32)],
         [(2, 2), (35, 35), (1000, 20)],
         [(1300, 1200)] + [(200 + i, 1) for i in range(20)]]


@pytest.mark.parametrize("segs", CASES)
@pytest.mark.parametrize("HQ,HKV,D,page_size,window,chunk", [(8, 2, 32, 16, None, 0), (4, 4, 64, 8, None, 0), (4, 2, 128, 16, None, 0),
                                                             (8, 8, 128, 16, None, 0), (3, 1, 128, 5, None, 0), (4, 2, 128, 16, 50, 0),
                                                             (2, 2, 64, 16, None, 48)])
def test_float32_attention_adds_in_the_plain_kernels_order(segs, HQ, HKV, D, page_size, window, chunk):
    from purhie_b200.csrc import ops
    case = paged_case(segs, HQ, HKV, D, page_size, torch.float32, seed=3)
    outs = []
    for q in (case["q"], off_by_one(case["q"])):
        out = torch.full((case["T"], HQ * D), float("nan"), device=DEV)
        ops.attention_generic(q, case["k_base"], case["v_base"], case["page_stride"], page_size, case["table"], case["row_seg"],
                              case["positions"], out, num_heads=HQ, num_kv_heads=HKV, head_dim=D, window=window,
                              scale=1.0 / math.sqrt(D), chunk=chunk)
        outs.append(out)
    assert not torch.isnan(outs[0]).any()
    assert torch.equal(outs[0], outs[1])


def attend(case, q, HQ, HKV, D, page_size=16):
    from purhie_b200.csrc import ops
    out = torch.full((case["T"], HQ * D), float("nan"), device=DEV)
    ops.attention_generic(q, case["k_base"], case["v_base"], case["page_stride"], page_size, case["table"], case["row_seg"],
                          case["positions"], out, num_heads=HQ, num_kv_heads=HKV, head_dim=D, window=None, scale=1.0 / math.sqrt(D))
    return out


# more rows than 32, none or few of them in portions long enough for tiles: decoded tokens alone, portions of three, both
# beside a prompt; more leftover rows than CTAs a head, and searches over several blocks of 128 tokens
SHORT = [[(200 - i % 7, 1) for i in range(512)], [(100, 3)] * 256, [(90, 70)] + [(60 + i, 1) for i in range(300)] + [(40, 3)] * 31,
         [(33 + i, 1) for i in range(33)], [(200, 2), (300, 257), (50, 3), (400, 131), (3, 1)]]


@pytest.mark.parametrize("segs", SHORT)
@pytest.mark.parametrize("HQ,HKV,D", [(1, 1, 128), (4, 2, 32), (16, 8, 64)])
def test_rows_that_tiles_leave_add_in_the_plain_kernels_order(segs, HQ, HKV, D):
    case = paged_case(segs, HQ, HKV, D, 16, torch.float32, seed=8)
    out, plain = attend(case, case["q"], HQ, HKV, D), attend(case, off_by_one(case["q"]), HQ, HKV, D)
    assert not torch.isnan(out).any() and torch.equal(out, plain)


@pytest.mark.parametrize("segs", SHORT[:2])
@pytest.mark.parametrize("HQ,HKV,D", [(2, 2, 64), (4, 2, 32)])
def test_rows_that_tiles_leave_are_not_slower_than_in_the_plain_kernel(segs, HQ, HKV, D):
    """Few heads and hundreds of short portions: 16 CTAs a head once took up to 2.4 times the plain kernel's time."""
    case = paged_case(segs, HQ, HKV, D, 16, torch.float32, seed=8)
    times = []
    for q in (case["q"], off_by_one(case["q"])):
        best = math.inf
        for _ in range(5):
            start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            start.record()
            for _ in range(4):
                attend(case, q, HQ, HKV, D)
            end.record()
            end.synchronize()
            best = min(best, start.elapsed_time(end))
        times.append(best)
    assert times[0] < times[1]


@pytest.mark.parametrize("cap", [0.0, 2.0])
@pytest.mark.parametrize("D", [32, 128])
def test_float32_attention_with_sink_bias_gate_and_cap(D, cap):
    from purhie_b200.csrc import ops
    HQ, HKV, ps = 4, 2, 16
    case = paged_case([(70, 40), (1, 1), (200, 1)], HQ, HKV, D, ps, torch.float32, seed=4)
    sink, slopes, gate = rnd(HQ, seed=5), rnd(HQ, seed=6).abs() * 0.05, rnd(case["T"], HQ * D, seed=7)
    if cap:
        slopes = None
    outs = []
    for q in (case["q"], off_by_one(case["q"])):
        out = torch.full((case["T"], HQ * D), float("nan"), device=DEV)
        ops.call("core", "ph_attention_generic_capped", ops._ptr(q), ops._code(q.dtype), ops._ptr(case["k_base"]), ops._ptr(case["v_base"]),
                 ops._code(torch.float32), case["page_stride"], ps, ops._ptr(case["table"]), case["table"].stride(0), ops._ptr(case["row_seg"]),
                 ops._ptr(case["positions"]), ops._ptr(out), ops._code(torch.float32), case["T"], HQ, HKV, D, 0, 1.0 / math.sqrt(D), D, 0, 0,
                 ops._ptr(sink), ops._ptr(slopes) if slopes is not None else None, ops._ptr(gate), HQ * D, cap, ops._stream())
        outs.append(out)
    assert not torch.isnan(outs[0]).any()
    assert torch.equal(outs[0], outs[1])


def product_us(M, N, K, dtype=torch.float32):
    """Time of one product among twenty in a graph, the weights in turn."""
    from purhie_b200.csrc import ops
    x, y = rnd(M, K, seed=1).to(dtype), torch.empty(M, N, device="cuda", dtype=dtype)
    ws = [rnd(N, K, seed=2).to(dtype) for _ in range(4)]
    ops.gemm_simple(x, ws[0], y)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        for i in range(20):
            ops.gemm_simple(x, ws[i % 4], y)
    best = float("inf")
    for _ in range(6):
        start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        start.record()
        graph.replay()
        end.record()
        end.synchronize()
        best = min(best, start.elapsed_time(end) * 50.0)
    return best


@pytest.mark.parametrize("M,N", [(8, 2048), (16, 2368)])
def test_short_products_of_more_columns_than_a_round_holds_are_not_shared_out(M, N):
    """Half of K takes 0.59 and 0.47 of the time as a chain a thread, 0.78 and 0.74 with K shared out in two rounds."""
    assert product_us(M, N, 384) < 0.68 * product_us(M, N, 768)


def test_tiles_of_one_group_where_their_number_an_sm_is_even():
    """Fourteen tiles an SM take as long as thirteen with one group a tile, 1.07 times as long with two."""
    assert product_us(2048, 1024, 3072) < 1.035 * product_us(1920, 1024, 3072)


def test_the_plain_kernel_waits_for_little_else_than_its_products():
    """One row of a weight whose K no fast kernel takes: 0.31 of the time of 512 rows, 0.58 with a wait for memory at every 16 of K."""
    assert product_us(1, 4096, 1020, torch.bfloat16) < 0.45 * product_us(512, 4096, 1020, torch.bfloat16)
