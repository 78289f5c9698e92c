"""Each kernel alone against its plain function (tests/plain_ops.py), at sizes other than the engine's."""
from __future__ import annotations

import numpy as np
import pytest
import torch

import plain_ops

pytestmark = pytest.mark.gpu

DTYPES = [torch.float32, torch.bfloat16]


def _tol(dtype, scale=1.0):
    return (2e-6 if dtype == torch.float32 else 1.6e-2) * scale


@pytest.fixture(scope="module")
def ops():
    from tinyllama_inference_engine_b200 import ops as module

    assert torch.cuda.is_available(), "these tests need the GPU"
    module.core()
    return module


def _paged_case(rng, dtype, seq_lens, q_lens, kv_heads, head_dim, page_size, q_heads):
    """Random cache pages for requests of ``seq_lens`` tokens, the last ``q_lens`` of which are this step's rows."""
    num_pages = sum(-(-s // page_size) for s in seq_lens) + 3
    order = rng.permutation(num_pages)
    width = max(-(-s // page_size) for s in seq_lens) + 1
    table = -np.ones((len(seq_lens), width), dtype=np.int32)
    at = 0
    for i, s in enumerate(seq_lens):
        n = -(-s // page_size)
        table[i, :n] = order[at : at + n]
        at += n
    pages = (torch.randn(num_pages, 2, kv_heads, page_size, head_dim) * 0.5).to(dtype)
    positions, token_seq = [], []
    for i, (s, q) in enumerate(zip(seq_lens, q_lens)):
        positions += list(range(s - q, s))
        token_seq += [i] * q
    tokens = len(positions)
    qkv = (torch.randn(tokens, (q_heads + 2 * kv_heads) * head_dim) * 0.5).to(dtype)
    return qkv, pages, torch.tensor(positions, dtype=torch.int32), torch.tensor(token_seq, dtype=torch.int32), torch.from_numpy(table)


@pytest.mark.parametrize("dtype", DTYPES)
def test_embedding(ops, dtype):
    torch.manual_seed(0)
    table = torch.randn(131, 80).to(dtype)
    ids = torch.tensor([0, 130, 5, 5, 77], dtype=torch.int32)
    want = torch.empty(5, 80)
    plain_ops.embedding(table, ids, want)
    got = torch.empty(5, 80, device="cuda")
    ops.embedding(table.cuda(), ids.cuda(), got)
    assert torch.equal(got.cpu(), want)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("hidden,eps", [(80, 1e-4), (2048, 1e-5), (1000, 1e-6)])
def test_add_rmsnorm(ops, dtype, hidden, eps):
    torch.manual_seed(1)
    residual = torch.randn(7, hidden) * 3
    delta = torch.randn(7, hidden).to(dtype)
    weight = 1 + 0.1 * torch.randn(hidden)
    for use_delta, rows in ((True, None), (False, None), (False, torch.tensor([6, 0, 3], dtype=torch.int32))):
        r_plain, r_gpu = residual.clone(), residual.clone().cuda()
        n = 7 if rows is None else 3
        want = torch.empty(n, hidden, dtype=dtype)
        plain_ops.add_rmsnorm(r_plain, delta if use_delta else None, weight, eps, want, rows)
        got = torch.empty(n, hidden, dtype=dtype, device="cuda")
        ops.add_rmsnorm(r_gpu, delta.cuda() if use_delta else None, weight.cuda(), eps, got, None if rows is None else rows.cuda())
        assert torch.allclose(r_gpu.cpu(), r_plain, atol=1e-6)
        assert torch.allclose(got.cpu().float(), want.float(), atol=_tol(dtype, 8), rtol=_tol(dtype))


@pytest.mark.parametrize("hidden", [2048, 1000, 4096, 5120])
def test_add_rmsnorm_of_many_rows(ops, hidden):
    """Steps of hundreds of rows normalise with a warp per row (bfloat16 out; widths up to 4096, wider ones on the other kernel)."""
    torch.manual_seed(2)
    rows_total, eps = 300, 1e-5
    residual = torch.randn(rows_total, hidden) * 3
    delta = torch.randn(rows_total, hidden).bfloat16()
    weight = 1 + 0.1 * torch.randn(hidden)
    picked = torch.randperm(rows_total)[:260].to(torch.int32)
    for use_delta, rows in ((True, None), (False, None), (False, picked)):
        r_plain, r_gpu = residual.clone(), residual.clone().cuda()
        n = rows_total if rows is None else rows.shape[0]
        want = torch.empty(n, hidden, dtype=torch.bfloat16)
        plain_ops.add_rmsnorm(r_plain, delta if use_delta else None, weight, eps, want, rows)
        got = torch.full((n, hidden), float("nan"), dtype=torch.bfloat16, device="cuda")
        ops.add_rmsnorm(r_gpu, delta.cuda() if use_delta else None, weight.cuda(), eps, got, None if rows is None else rows.cuda())
        assert torch.allclose(r_gpu.cpu(), r_plain, atol=1e-6)
        assert torch.allclose(got.cpu().float(), want.float(), atol=_tol(torch.bfloat16, 8), rtol=_tol(torch.bfloat16))


@pytest.mark.parametrize("dtype", DTYPES)
def test_silu_mul_and_add(ops, dtype):
    torch.manual_seed(2)
    gate_up = (torch.randn(5, 2 * 176) * 2).to(dtype)
    want = torch.empty(5, 176, dtype=dtype)
    plain_ops.silu_mul(gate_up, want)
    got = torch.empty(5, 176, dtype=dtype, device="cuda")
    ops.silu_mul(gate_up.cuda(), got)
    assert torch.allclose(got.cpu().float(), want.float(), atol=_tol(dtype, 4), rtol=_tol(dtype))
    residual = torch.randn(5, 176)
    delta = torch.randn(5, 176).to(dtype)
    r = residual.clone().cuda()
    ops.add_(r, delta.cuda())
    assert torch.allclose(r.cpu(), residual + delta.float(), atol=1e-6)


@pytest.mark.parametrize("M,N,K", [(1, 256, 64), (37, 131, 80), (130, 70, 513), (3, 1000, 17)])
def test_gemm_fp32_is_true_32_bit(ops, M, N, K):
    torch.manual_seed(3)
    x, w = torch.randn(M, K), torch.randn(N, K)
    want = (x.double() @ w.double().T).float()
    got = torch.empty(M, N, device="cuda")
    ops.linear(x.cuda(), w.cuda(), got)
    # a reduced-precision (tf32 / bf16) product would be off by ~1e-3 * sqrt(K) here
    assert torch.allclose(got.cpu(), want, atol=2e-6 * K ** 0.5 * 4, rtol=1e-6)
    # one row alone gives bit-identical numbers: the order of a row's sum does not depend on the batch
    alone = torch.empty(1, N, device="cuda")
    ops.linear(x[M - 1 :].cuda(), w.cuda(), alone)
    assert torch.equal(alone[0], got[M - 1])


def _error(got, x, w) -> float:
    """Against 64-bit sums, 2-norms."""
    exact = x.double() @ w.double().T
    return float((got.double() - exact).norm() / exact.norm())


def _parts_limit(K: int) -> float:
    """Chunks of 64 k are added in order, one rounding of at most 2^-24 each of a sum that grows with the root of their number, and 2^-24 for what happens inside a chunk.  (Measured: 0.75e-7 at one
    chunk, 1.3e-7 at 32, 1.9e-7 at 88.  A sum of multiply-adds in order is off by 8.1e-7 at K = 2,048, parts without middle times middle by about 3e-6, bfloat16 operands by 2e-3.)"""
    return 2.0 ** -24 * ((-(-K // 64) / 2) ** 0.5 + 1)


@pytest.mark.parametrize("M,N", [(1, 2048), (8, 5000), (16, 2048), (64, 2048), (256, 2048), (600, 3000)])
@pytest.mark.parametrize("K", [64, 512, 2048, 5632])
def test_gemm_fp32_is_nearer_to_64_bits_than_a_sum_in_order(ops, M, N, K):
    """Blocks of 8 and 16 rows, tiles of 128 x 64 and of 128 x 96."""
    torch.manual_seed(62)
    x, w = torch.randn(M, K).cuda(), torch.randn(N, K).cuda()
    got = torch.empty(M, N, device="cuda")
    ops.linear(x, w, got)
    assert _error(got, x, w) <= _parts_limit(K)


@pytest.mark.parametrize("K", [130, 260, 2048])
@pytest.mark.parametrize("kind", ["spread", "cancelling", "sparse"])
def test_gemm_fp32_gives_uneven_terms_the_same_bits_in_every_kernel(ops, kind, K):
    """Blocks of rows run on mma.sync and tiles on tcgen05.  Terms over 2^-60 to 2^60, terms that cancel but for their last bits, and rows of mostly zeros, where an order of sums shows."""
    torch.manual_seed(63)
    M, N = 300, 2050
    x, w = torch.randn(M, K), torch.randn(N, K)
    if kind == "spread":
        x *= 2.0 ** torch.randint(-30, 31, (M, K))
        w *= 2.0 ** torch.randint(-30, 31, (N, K))
    elif kind == "cancelling":
        half = K // 2
        order = torch.randperm(half)
        x[:, half : 2 * half], w[:, half : 2 * half] = -x[:, order] * (1 + 2.0 ** -20), w[:, order]
    else:
        x *= torch.rand(M, K) < 0.1
        w *= torch.rand(N, K) < 0.3
    x, w = x.cuda(), w.cuda()
    full = torch.empty(M, N, device="cuda")
    ops.linear(x, w, full)
    bound = K * 2.0 ** -24 * (x.double().abs() @ w.double().abs().T)
    assert bool(((full.double() - x.double() @ w.double().T).abs() <= bound).all())
    for first, rows in ((0, 1), (5, 8), (17, 16), (100, 16), (250, 40), (284, 16)):
        got = torch.empty(rows, N, device="cuda")
        ops.linear(x[first : first + rows], w, got)
        assert torch.equal(got, full[first : first + rows]), (first, rows)


@pytest.mark.parametrize("N,K", [(64, 128), (130, 516), (2049, 260), (16, 4)])
def test_gemm_fp32_gives_a_row_the_same_bits_in_every_kernel(ops, N, K):
    """Blocks of 8 and 16 rows, tiles of 128 rows and, with an operand that is not 16-byte aligned, their forms with 4-byte copies; four terms: the kernel of short sums."""
    torch.manual_seed(33)
    x, w = torch.randn(900, K).cuda(), torch.randn(N, K).cuda()
    full = torch.empty(900, N, device="cuda")
    ops.linear(x, w, full)
    # one rounding per multiply-add of a sum of K terms
    bound = K * 2.0 ** -24 * (x.double().abs() @ w.double().abs().T)
    assert bool(((full.double() - x.double() @ w.double().T).abs() <= bound).all())
    assert _error(full, x, w) <= _parts_limit(K)
    for M in (1, 2, 3, 4, 5, 8, 9, 16, 17, 31, 33, 64, 65, 129, 300):
        got = torch.full((M, N), float("nan"), device="cuda")
        ops.linear(x[7 : 7 + M], w, got)
        assert torch.equal(got, full[7 : 7 + M]), M
    wide = torch.randn(40, K + 1).cuda()   # rows one element apart from 16-byte alignment: 4-byte copies
    wide[:, :K] = x[:40]
    got = torch.empty(40, N, device="cuda")
    ops.linear(wide[:, :K], w, got)
    assert torch.equal(got, full[:40])


@pytest.mark.parametrize("N,K", [(96, 6208), (97, 64), (200, 14404), (2048, 36), (161, 130), (2050, 130), (2081, 6212)])   # the last two are wide enough for tiles from 129 rows on, the others mostly blocks of 16
def test_gemm_fp32_in_parts_around_tiles_and_rounds(ops, N, K):
    """Tiles of 128 rows of x by 64 or 96 of w, chunks of 64 k, rounds of 96 chunks, 16-byte copies and 4-byte ones: against 64-bit sums, and every row with the bits it has alone."""
    torch.manual_seed(53)
    x, w = torch.randn(600, K).cuda(), torch.randn(N, K).cuda()
    exact = x.double() @ w.double().T
    bound = K * 2.0 ** -24 * (x.double().abs() @ w.double().abs().T)   # one rounding per multiply-add of a sum of K terms: what a sum in order is held to
    alone = torch.empty(600, N, device="cuda")
    for first in range(0, 600, 16):
        ops.linear(x[first : first + 16], w, alone[first : first + 16])
    assert bool(((alone.double() - exact).abs() <= bound).all()) and _error(alone, x, w) <= _parts_limit(K)
    for M in (17, 63, 127, 128, 129, 256, 257, 600):
        got = torch.full((M, N), float("nan"), device="cuda")
        ops.linear(x[:M], w, got)
        assert torch.equal(got, alone[:M]), M
    assert int(ops.error_flag(x.device)) == 0, "a bounded wait inside the kernel gave up"


@pytest.mark.parametrize("M", [1, 12, 140])
def test_gemm_fp32_of_numbers_whose_parts_fall_out_of_range(ops, M):
    """Infinities, NaN, sums beyond the largest number, numbers near it, and results near the smallest: as one sum of multiply-adds gives them."""
    torch.manual_seed(54)
    N, K = 100, 132
    x, w = torch.randn(M, K), torch.randn(N, K)
    w[:, 1] = 1.0   # (its middle and low parts are 0)
    x[0, 1] = float("inf")
    w[3, 5] = float("-inf")
    w[7, 9] = float("nan")
    w[11] = 3.3e38                      # sums beyond the largest number
    w[12] = 0.0
    w[12, 20] = 3.4028234e38            # its leading part would round to infinity
    w[13] *= 1e-38                      # parts below the smallest bfloat16
    x[:, 20] = 0.5
    got = torch.empty(M, N, device="cuda")
    ops.linear(x.cuda(), w.cuda(), got)
    want = torch.zeros(M, N)
    for k in range(K):   # (a product is exact in 64 bits, so one rounding to 32 bits per step, as a multiply-add's, but for ties of two roundings)
        want = (want.double() + x[:, k].double()[:, None] * w[:, k].double()[None, :]).float()
    got = got.cpu()
    assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got.isinf(), want.isinf())
    assert torch.equal(got[want.isinf()], want[want.isinf()])
    finite = want.isfinite()
    bound = K * 2.0 ** -23 * (x.double().abs() @ w.double().abs().T) + K * 2.0 ** -149
    assert bool(((got.double() - want.double()).abs() <= bound)[finite].all())


@pytest.mark.parametrize("M", [4, 12, 300])
@pytest.mark.parametrize("K", [131, 132, 1000])
def test_gemm_fp32_beside_infinities_and_nan(ops, M, K):
    """Rows of x and of w with an infinity, a NaN, zeros or large numbers, in the few-rows kernel and in tiles: their outputs are sums in order, all others have the bits they have without them."""
    torch.manual_seed(58)
    N = 2050
    x, w = torch.randn(M, K), torch.randn(N, K)
    plain = torch.empty(M, N, device="cuda")
    ops.linear(x.cuda(), w.cuda(), plain)
    special = {"inf": (0, 3), "nan": (1, 100), "zero": (2, 1030), "large": (M - 1, 2049)}
    for kind, (m, n) in special.items():
        for row in (x[m], w[n]):
            if kind == "zero":
                row.zero_()
            elif kind == "large":
                row *= 1e17
            else:
                row[K // 2 + (n & 1)] = float(kind)
    got = torch.full((M, N), -1.0, device="cuda")
    ops.linear(x.cuda(), w.cuda(), got)
    got, plain = got.cpu(), plain.cpu()
    rows, columns = [m for m, _ in special.values()], [n for _, n in special.values()]
    others_m, others_n = [m for m in range(M) if m not in rows], [n for n in range(N) if n not in columns]
    assert torch.equal(got[others_m][:, others_n], plain[others_m][:, others_n])
    exact = x.double() @ w.double().T
    want = torch.zeros(M, N)
    for k in range(K):
        want = (want.double() + x[:, k].double()[:, None] * w[:, k].double()[None, :]).float()
    assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got[want.isinf()], want[want.isinf()]) and bool((got[2] == 0)[~want[2].isnan()].all())
    bound = K * 2.0 ** -24 * (x.double().abs() @ w.double().abs().T)
    assert bool(((got.double() - exact).abs() <= bound)[want.isfinite()].all())
    assert int(ops.error_flag(torch.device("cuda", 0))) == 0, "a bounded wait inside the kernel gave up"


def test_gemm_fp32_with_a_nan_takes_a_few_times_as_long_at_most(ops):
    """A NaN settles its outputs and an infinity's are summed by the whole tile (2.4 and 6 times the product's time, measured; one thread for a row of a tile's outputs took 80 times)."""
    torch.manual_seed(59)
    x, w, out = torch.randn(760, 2048).cuda(), torch.randn(2048, 2048).cuda(), torch.empty(760, 2048, device="cuda")

    def fastest():
        times = []
        for _ in range(6):
            start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            start.record()
            for _ in range(4):
                ops.linear(x, w, out)
            end.record()
            torch.cuda.synchronize()
            times.append(start.elapsed_time(end))
        return min(times)

    without = fastest()
    for value in (float("nan"), float("inf")):
        x[5, 7] = value
        assert fastest() < 20 * without, value


@pytest.mark.parametrize("K", [7, 63, 64, 65, 128, 130, 192, 200, 256, 260])
def test_gemm_fp32_of_short_rows(ops, K):
    """Warps take chunks of several tiles at a time where a row has one to four of them (and one tile at a time above): the bits of the tiles of 128 rows, also beside outputs that are worked out again."""
    torch.manual_seed(61)
    N = 11290   # more tiles of 16 than CTAs, the last of them and the last group of tiles not full
    x, w = torch.randn(300, K).cuda(), torch.randn(N, K).cuda()
    exact = x.double() @ w.double().T
    full = torch.empty(300, N, device="cuda")
    ops.linear(x, w, full)
    assert bool(((full.double() - exact).abs() <= K * 2.0 ** -24 * (x.double().abs() @ w.double().abs().T)).all())
    again = w.clone()
    again[40], again[4800], again[11288] = float("nan"), again[4800] * 1e-37, float("inf")
    worked = torch.empty(300, N, device="cuda")
    ops.linear(x, again, worked)
    plain = torch.ones(N, dtype=torch.bool)
    plain[[40, 4800, 11288]] = False
    assert torch.equal(worked[:, plain], full[:, plain])
    for M in (1, 5, 8, 9, 16, 24, 40):
        for weight, want in ((w, full), (again, worked)):
            got = torch.full((M, N), float("nan"), device="cuda")
            ops.linear(x[11 : 11 + M], weight, got)
            assert torch.equal(got.view(torch.int32), want[11 : 11 + M].view(torch.int32)), M
    wide = torch.randn(8, K + 1).cuda()
    wide[:, :K] = x[:8]
    got = torch.empty(8, N, device="cuda")
    ops.linear(wide[:, :K], w, got)   # 4-byte copies
    assert torch.equal(got, full[:8])


TINY_AND_LARGE = [(1e3, 1e-33), (1e5, 1e-35), (1e8, 1e-36), (1e9, 2e-38), (1e20, 2e-41), (1e10, 1e-43)]


@pytest.mark.parametrize("K", [64, 130])
@pytest.mark.parametrize("M", [4, 12, 300])
@pytest.mark.parametrize("sx,sw", TINY_AND_LARGE + [pair[::-1] for pair in TINY_AND_LARGE])
def test_gemm_fp32_of_tiny_numbers_times_large_ones(ops, sx, sw, M, K):
    """Results far above the smallest number whose terms have an operand near it or below (of which three bfloat16 parts hold few bits or none)."""
    torch.manual_seed(55)
    N = 2050
    x, w = (torch.randn(M, K, dtype=torch.float64) * sx).float().cuda(), (torch.randn(N, K, dtype=torch.float64) * sw).float().cuda()
    x[1], w[5] = 0.0, 0.0
    exact = x.double() @ w.double().T
    got = torch.full((M, N), float("nan"), device="cuda")
    ops.linear(x, w, got)
    # a sum of K terms in order, one rounding of at most 2^-24 per step of what has grown with the root of the step, is off by 2^-24 sqrt(K / 2) at most (2-norms)
    assert float((got.double() - exact).norm() / exact.norm()) <= 2.0 ** -24 * (K / 2) ** 0.5
    assert bool((got[1] == 0).all()) and bool((got[:, 5] == 0).all())


@pytest.mark.parametrize("M", [1, 17, 300])
@pytest.mark.parametrize("K", [1, 2, 3, 4, 5, 6])
def test_gemm_fp32_of_a_few_terms_is_their_sum_in_order(ops, K, M):
    """A single product is the rounded one, and every multiply-add after it rounds once: the bits of a sum in order."""
    torch.manual_seed(57)
    N = 2050
    x, w = torch.randn(M, K), torch.randn(N, K)
    want = torch.zeros(M, N, dtype=torch.float64)
    ties = torch.zeros(M, N, dtype=torch.bool)   # where the 64-bit sum is itself rounded, a tie of 32-bit numbers may fall on the other side
    for k in range(K):
        step = want + x[:, k].double()[:, None] * w[:, k].double()[None, :]
        ties |= (step.float().double() - step).abs() == (torch.nextafter(step.float(), torch.where(step.float().double() < step, 1.0, -1.0) * float("inf")).double() - step).abs()
        want = step.float().double()
    got = torch.empty(M, N, device="cuda")
    ops.linear(x.cuda(), w.cuda(), got)
    assert int(ties.sum()) <= 4 and torch.equal(got.cpu()[~ties], want.float()[~ties])


@pytest.mark.parametrize("M", [4, 12, 300])
def test_gemm_fp32_gives_a_row_its_bits_beside_rows_of_tiny_numbers(ops, M):
    """Whether an output is worked out again is a matter of its own two rows: neighbours in its tile change nothing, nor do other rows of its product."""
    torch.manual_seed(56)
    N, K = 2050, 260
    x, w = torch.randn(M, K).cuda(), torch.randn(N, K).cuda()
    plain = torch.empty(M, N, device="cuda")
    ops.linear(x, w, plain)
    w[::3] *= 1e-37
    w[1, 7] = 1e-41   # a normal row with one number that its parts do not hold: lost in what its sums round off
    x[3] *= 1e-30
    got = torch.empty(M, N, device="cuda")
    ops.linear(x, w, got)
    kept = [m for m in range(M) if m != 3]
    columns = [n for n in range(N) if n % 3 and n != 1]
    assert torch.equal(got[kept][:, columns], plain[kept][:, columns])
    alone = torch.empty(1, N, device="cuda")
    for m in (0, 2, 3, M - 1):
        ops.linear(x[m : m + 1], w, alone)
        assert torch.equal(alone[0], got[m]), m
    exact = x.double() @ w.double().T
    bound = K * 2.0 ** -24 * (x.double().abs() @ w.double().abs().T) + K * 2.0 ** -149
    assert bool(((got.double() - exact).abs() <= bound).all())


@pytest.mark.parametrize("M", [1, 2, 4, 8, 16, 40])
def test_gemm_fp32_takes_a_weight_that_the_kernel_before_it_writes(ops, M):
    """A product whose weight is the result of the product before it (which lets its successor start early), over and over on the same buffer."""
    torch.manual_seed(38)
    N, K = 1000, 2048
    a, b, x = torch.randn(3, N, 256).cuda(), torch.randn(K, 256).cuda(), torch.randn(M, K).cuda()
    weight, out = torch.zeros(N, K, device="cuda"), torch.zeros(3, M, N, device="cuda")
    want = torch.zeros_like(out)
    for i in range(3):
        ops.linear(a[i], b, weight)
        torch.cuda.synchronize()
        ops.linear(x, weight, want[i])
        torch.cuda.synchronize()
    for _ in range(5):
        for i in range(3):
            ops.linear(a[i], b, weight)
            ops.linear(x, weight, out[i])
        assert torch.equal(out, want)


@pytest.mark.parametrize("M,K", [(1, 2048), (4, 2048), (16, 2048), (40, 2048), (400, 2048), (4, 2046), (400, 2046)])
def test_gemm_fp32_takes_activations_that_the_kernel_before_it_writes(ops, M, K):
    """The same with x, the result of the product before it: every chunk of it has to be what was written last, whatever an earlier product on the same buffer left in a cache."""
    torch.manual_seed(60)
    N = 1100
    a, b, w = torch.randn(3, M, 256).cuda(), torch.randn(K, 256).cuda(), torch.randn(N, K).cuda()
    x, out = torch.zeros(M, K, device="cuda"), torch.zeros(3, M, N, device="cuda")
    want = torch.zeros_like(out)
    for i in range(3):
        ops.linear(a[i], b, x)
        torch.cuda.synchronize()
        ops.linear(x, w, want[i])
        torch.cuda.synchronize()
    for _ in range(5):
        for i in range(3):
            ops.linear(a[i], b, x)
            ops.linear(x, w, out[i])
        assert torch.equal(out, want)


@pytest.mark.parametrize("M,N,K", [(1, 256, 64), (37, 136, 80), (130, 72, 520), (64, 2048, 2048)])
def test_linear_bf16(ops, M, N, K):
    torch.manual_seed(4)
    x, w = torch.randn(M, K).bfloat16(), torch.randn(N, K).bfloat16()
    want = x.float() @ w.float().T
    got = torch.empty(M, N, dtype=torch.bfloat16, device="cuda")
    ops.linear(x.cuda(), w.cuda(), got)
    assert torch.allclose(got.cpu().float(), want, atol=1e-2 * K ** 0.5, rtol=1e-2)
    got32 = torch.empty(M, N, dtype=torch.float32, device="cuda")
    ops.linear(x.cuda(), w.cuda(), got32)
    assert torch.allclose(got32.cpu(), want, atol=2e-5 * K ** 0.5, rtol=1e-5)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("q_heads,kv_heads,head_dim,page_size,rotary_dim,theta", [(4, 2, 16, 16, 16, 1e4), (6, 2, 32, 32, 32, 5e5), (3, 3, 48, 16, 24, 777.0), (8, 1, 128, 64, 128, 1e4),
                                                                             (5, 1, 64, 16, 32, 1e4)])
def test_rope_store(ops, dtype, q_heads, kv_heads, head_dim, page_size, rotary_dim, theta):
    rng = np.random.default_rng(5)
    torch.manual_seed(5)
    seq_lens, q_lens = [4100, 17, page_size + 1, 1], [5, 17, 2, 1]
    qkv, pages, positions, token_seq, table = _paged_case(rng, dtype, seq_lens, q_lens, kv_heads, head_dim, page_size, q_heads)
    exponent = (np.float32(-2.0) * np.arange(rotary_dim // 2, dtype=np.float32)) / np.float32(rotary_dim)
    inv_freq = torch.from_numpy(np.power(np.float32(theta), exponent, dtype=np.float32))
    for write in (True, False):
        qkv_plain, pages_plain = qkv.clone(), pages.clone()
        plain_ops.rope_store(qkv_plain, positions, token_seq, table, inv_freq, rotary_dim, pages_plain, q_heads, kv_heads, head_dim, page_size, write)
        qkv_gpu, pages_gpu = qkv.clone().cuda(), pages.clone().cuda()
        ops.rope_store(qkv_gpu, positions.cuda(), token_seq.cuda(), table.cuda(), inv_freq.cuda(), rotary_dim, pages_gpu, q_heads, kv_heads, head_dim, page_size, write)
        q_width = q_heads * head_dim
        # position 4099 with 32-bit angles: sine and cosine of the two sides may differ in the last bits
        assert torch.allclose(qkv_gpu.cpu().float()[:, :q_width], qkv_plain.float()[:, :q_width], atol=_tol(dtype, 4) + 2e-4)
        assert torch.equal(qkv_gpu.cpu()[:, q_width:], qkv_plain[:, q_width:])
        assert torch.allclose(pages_gpu.cpu().float(), pages_plain.float(), atol=_tol(dtype, 4) + 2e-4)
        if not write:
            assert torch.equal(pages_gpu.cpu(), pages)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("q_heads,kv_heads,head_dim,page_size,window", [(4, 2, 16, 16, 0), (6, 2, 32, 32, 0), (3, 3, 48, 16, 0), (8, 1, 128, 64, 0), (4, 4, 80, 16, 0), (4, 2, 64, 16, 37), (32, 4, 64, 64, 0)])
def test_paged_attention(ops, dtype, q_heads, kv_heads, head_dim, page_size, window):
    rng = np.random.default_rng(6)
    torch.manual_seed(6)
    seq_lens = [300, page_size, page_size + 1, 1, 2 * page_size - 1, 131]
    q_lens = [7, page_size, 2, 1, 1, 131]
    qkv, pages, positions, token_seq, table = _paged_case(rng, dtype, seq_lens, q_lens, kv_heads, head_dim, page_size, q_heads)
    # one far key among hundreds: make a single early key of request 0 match its last query strongly
    q_row = sum(q_lens[:1]) - 1
    page, slot = int(table[0, 3 // page_size]), 3 % page_size
    for h in range(q_heads):
        qv = qkv.view(qkv.shape[0], -1, head_dim)[q_row, h].float()
        pages[page, 0, h // (q_heads // kv_heads), slot] = (qv * (6.0 / max(1e-3, float(qv.norm()) ** 2) * head_dim ** 0.5)).to(dtype)
    tokens = qkv.shape[0]
    want = torch.empty(tokens, q_heads * head_dim, dtype=dtype)
    plain_ops.paged_attention(qkv, pages, positions, token_seq, table, want, q_heads, kv_heads, head_dim, page_size, window)
    got = torch.empty(tokens, q_heads * head_dim, dtype=dtype, device="cuda")
    ops.paged_attention(qkv.cuda(), pages.cuda(), positions.cuda(), token_seq.cuda(), table.cuda(), got, q_heads, kv_heads, head_dim, page_size, window)
    assert torch.allclose(got.cpu().float(), want.float(), atol=_tol(dtype, 2) + (2e-6 if dtype == torch.float32 else 0)), float((got.cpu().float() - want.float()).abs().max())


def test_embedding_survives_an_id_outside_the_table_and_reports_it(ops):
    """An id the host never saw (a token sampled on the device from non-finite logits) must not be used as an address:
    row 0 is read instead and the device's error word says so; reading the word raises and clears it."""
    from tinyllama_inference_engine_b200.errors import KernelError

    table = torch.randn(50, 64).bfloat16().cuda()
    ids = torch.tensor([3, 50, -1, 0x7FFFFFFF, 49], dtype=torch.int32).cuda()
    got = torch.empty(5, 64, device="cuda")
    ops.check_device_errors(got.device)   # nothing is pending
    ops.embedding(table, ids, got)
    with pytest.raises(KernelError, match="outside the vocabulary"):
        ops.check_device_errors(got.device)
    ops.check_device_errors(got.device)   # cleared by the read that raised
    want = table.float()[[3, 0, 0, 0, 49]]
    assert torch.equal(got, want)


@pytest.mark.parametrize("rows", [1, 3, 1023, 1024, 1027])
def test_rows_of_eight_at_a_time(ops, rows):
    """Embedding, gate and rotation in pieces of eight elements: widths of whole pieces and others, rotation with one token per block and with four."""
    torch.manual_seed(37)
    for width in (8, 2048, 2056, 2052, 131):
        table, ids = torch.randn(50, width).bfloat16(), torch.randint(0, 50, (rows,), dtype=torch.int32)
        got = torch.empty(rows, width, device="cuda")
        ops.embedding(table.cuda(), ids.cuda(), got)
        assert torch.equal(got.cpu(), table.float()[ids.long()])
        gate_up = torch.randn(rows, 2 * width).bfloat16()
        want, got = torch.empty(rows, width, dtype=torch.bfloat16), torch.empty(rows, width, dtype=torch.bfloat16, device="cuda")
        plain_ops.silu_mul(gate_up, want)
        ops.silu_mul(gate_up.cuda(), got)
        assert torch.allclose(got.cpu().float(), want.float(), atol=_tol(torch.bfloat16, 4), rtol=_tol(torch.bfloat16))
    rng = np.random.default_rng(37)
    qkv, pages, positions, token_seq, table = _paged_case(rng, torch.bfloat16, [rows], [rows], 2, 64, 64, 6)
    inv_freq = torch.from_numpy(np.power(np.float32(1e4), np.float32(-2.0) * np.arange(16, dtype=np.float32) / np.float32(32)))
    qkv_plain, pages_plain = qkv.clone(), pages.clone()
    plain_ops.rope_store(qkv_plain, positions, token_seq, table, inv_freq, 32, pages_plain, 6, 2, 64, 64, True)
    qkv_gpu, pages_gpu = qkv.clone().cuda(), pages.clone().cuda()
    ops.rope_store(qkv_gpu, positions.cuda(), token_seq.cuda(), table.cuda(), inv_freq.cuda(), 32, pages_gpu, 6, 2, 64, 64, True)
    assert torch.allclose(qkv_gpu.cpu().float(), qkv_plain.float(), atol=_tol(torch.bfloat16, 4) + 2e-4)
    assert torch.allclose(pages_gpu.cpu().float(), pages_plain.float(), atol=_tol(torch.bfloat16, 4) + 2e-4)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("hidden", [4, 40, 512, 516, 1024, 1028, 2048, 2050])
def test_embedding_of_narrow_and_wide_rows(ops, dtype, hidden):
    """Rows that share a block and rows that a block walks, numbers of rows that do not fill the last block, ids outside the table among them."""
    torch.manual_seed(43)
    table = torch.randn(50, hidden).to(dtype).cuda()
    for rows in (1, 3, 255, 257):
        ids = torch.randint(0, 50, (rows,), dtype=torch.int32)
        got = torch.full((rows + 1, hidden), 7.0, device="cuda")
        ops.embedding(table, ids.cuda(), got[:rows])
        assert torch.equal(got[:rows], table[ids.cuda().long()].float()) and bool((got[rows:] == 7.0).all())
    ids[5], ids[256] = -1, 50
    ops.embedding(table, ids.cuda(), got[:rows])
    with pytest.raises(Exception, match="outside the vocabulary"):
        ops.check_device_errors(got.device)
    assert torch.equal(got[5], table[0].float()) and torch.equal(got[256], table[0].float())


@pytest.mark.parametrize("inter", [8, 24, 120, 128, 136, 1016, 1032, 2048, 2056])
def test_gate_of_narrow_rows(ops, inter):
    """Rows that share a block (two to 256 of them) and rows that a block or two take, numbers of rows that do not fill the last block, both gates."""
    torch.manual_seed(42)
    for rows in (1, 3, 255, 257):
        gate_up = torch.randn(rows + 1, 2 * inter).bfloat16().cuda()
        g, u = gate_up[:rows, :inter].double(), gate_up[:rows, inter:].double()
        for kind, want in (("silu", g / (1 + torch.exp(-g)) * u), ("gelu_tanh", torch.nn.functional.gelu(g, approximate="tanh") * u)):
            got = torch.full((rows + 1, inter), 7.0, dtype=torch.bfloat16, device="cuda")
            ops.gate_mul(gate_up[:rows], got[:rows], kind)
            # one rounding to bfloat16 (2^-9 of the value) over 32-bit arithmetic
            assert bool(((got[:rows].double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-6).all()) and bool((got[rows:] == 7.0).all())


@pytest.mark.parametrize("q_heads,kv_heads,head_dim,rotary_dim", [(6, 2, 64, 32), (1, 1, 16, 16), (4, 4, 64, 64), (5, 1, 64, 64), (32, 32, 128, 128), (3, 2, 48, 0), (2, 2, 128, 80)])
@pytest.mark.parametrize("tokens", [2, 1023, 1025])
def test_rope_store_with_one_token_per_block_and_with_four(ops, q_heads, kv_heads, head_dim, rotary_dim, tokens):
    """Shapes on both sides of what decides between the two kernels (1,024 tokens; 64 pieces of a token), more pieces than threads, tails past the rotated part, no cache."""
    torch.manual_seed(40)
    qkv, pages, positions, token_seq, table = _paged_case(np.random.default_rng(40), torch.bfloat16, [tokens], [tokens], kv_heads, head_dim, 64, q_heads)
    inv_freq = torch.from_numpy(np.power(np.float32(1e4), np.float32(-2.0) * np.arange(rotary_dim // 2, dtype=np.float32) / np.float32(max(2, rotary_dim)))) if rotary_dim else None
    for write in (True, False):
        want_qkv, want_pages = qkv.clone(), pages.clone()
        plain_ops.rope_store(want_qkv, positions, token_seq, table, inv_freq, rotary_dim, want_pages, q_heads, kv_heads, head_dim, 64, write)
        got_qkv, got_pages = qkv.cuda(), pages.cuda()
        ops.rope_store(got_qkv, positions.cuda(), token_seq.cuda(), table.cuda(), None if inv_freq is None else inv_freq.cuda(), rotary_dim, got_pages, q_heads, kv_heads, head_dim, 64, write)
        assert torch.allclose(got_qkv.cpu().float(), want_qkv.float(), atol=_tol(torch.bfloat16, 4) + 2e-4)
        assert torch.allclose(got_pages.cpu().float(), want_pages.float(), atol=_tol(torch.bfloat16, 4) + 2e-4)


@pytest.mark.parametrize("tokens", [3, 500, 1500])
def test_rope_store_takes_positions_that_the_kernel_before_it_writes(ops, tokens):
    """Positions, rows' requests and block table gathered by a kernel that lets its successor start early, another choice of them each time."""
    torch.manual_seed(39)
    held = -(-tokens // 64)
    qkv, pages = torch.randn(tokens, 10 * 64).bfloat16(), torch.zeros(2 * held, 2, 2, 64, 64, dtype=torch.bfloat16)
    inv_freq = torch.from_numpy(np.power(np.float32(1e4), np.float32(-2.0) * np.arange(32, dtype=np.float32) / np.float32(64)))
    table = torch.randperm(2 * held)
    choices = torch.stack([torch.cat([torch.arange(tokens).roll(shift), torch.full((tokens,), shift % 2), table.roll(shift)]) for shift in range(4)]).int()
    described = torch.zeros(1, choices.shape[1], dtype=torch.int32, device="cuda")
    cut = lambda row: (row[:tokens], row[tokens : 2 * tokens], row[2 * tokens :].view(2, held))  # noqa: E731
    choices_gpu, freq = choices.cuda(), inv_freq.cuda()
    index = [torch.tensor([i], dtype=torch.int32, device="cuda") for i in range(4)]
    for i in (1, 3, 0, 2):
        want_qkv, want_pages = qkv.clone(), pages.clone()
        plain_ops.rope_store(want_qkv, *cut(choices[i]), inv_freq, 64, want_pages, 6, 2, 64, 64, True)
        for _ in range(3):
            got_qkv, got_pages = qkv.cuda(), pages.cuda()
            torch.cuda.synchronize()
            ops.gather_rows(choices_gpu, index[(i + 1) % 4], described)
            ops.gather_rows(choices_gpu, index[i], described)
            ops.rope_store(got_qkv, *cut(described[0]), freq, 64, got_pages, 6, 2, 64, 64, True)
            assert torch.allclose(got_qkv.cpu().float(), want_qkv.float(), atol=_tol(torch.bfloat16, 4) + 2e-4)
            assert torch.allclose(got_pages.cpu().float(), want_pages.float(), atol=_tol(torch.bfloat16, 4) + 2e-4)


@pytest.mark.parametrize("dtype,width", [(torch.float32, 2048), (torch.bfloat16, 4096), (torch.bfloat16, 131), (torch.float32, 3)])
def test_gather_rows(ops, dtype, width):
    x = torch.randn(40, width).to(dtype).cuda()
    for rows in ([39], [0, 7, 7, 3], list(range(39, -1, -1))):
        index = torch.tensor(rows, dtype=torch.int32).cuda()
        out = torch.empty(len(rows), width, dtype=dtype, device="cuda")
        ops.gather_rows(x, index, out)
        assert torch.equal(out, x[index.long()])


def test_sampling_non_finite_logits_still_gives_a_token_of_the_vocabulary(ops):
    vocab = 131
    logits = torch.randn(6, vocab)
    logits[0] = float("nan")
    logits[1] = float("-inf")
    logits[2, ::2] = float("nan")
    logits[3] = float("inf")
    logits[4, 5] = float("nan")
    cuda = lambda t: t.cuda()  # noqa: E731
    for temperature, top_p in ((0.0, 1.0), (0.9, 1.0), (0.9, 0.5)):
        out = torch.full((6,), -7, dtype=torch.int32, device="cuda")
        ops.sample(cuda(logits), cuda(torch.full((6,), temperature)), cuda(torch.full((6,), top_p)), cuda(torch.arange(6, dtype=torch.int64)),
                   cuda(torch.zeros(6, dtype=torch.int64)), out)
        tokens = out.cpu().tolist()
        assert all(0 <= t < vocab for t in tokens), (temperature, top_p, tokens)
    out = torch.full((6,), -7, dtype=torch.int32, device="cuda")
    ops.argmax(cuda(logits), out)
    assert all(0 <= t < vocab for t in out.cpu().tolist())


@pytest.mark.parametrize("vocab", [131, 4, 32000, 32772, 50304, 128256, 131076])
def test_greedy_rows_with_little_to_compare(ops, vocab):
    """Rows of NaN (token 0) and rows with one comparable value among NaN, read whole and in slices whose last loads are not full; both greedy kernels."""
    places = sorted({0, vocab // 4, vocab // 2 + 1, vocab - 1})
    logits = torch.full((1 + 2 * len(places) + 1, vocab), float("nan"))
    want = [0]
    for place in places:
        for value in (float("-inf"), -3.0):
            logits[len(want), place] = value
            want.append(place)
    logits[-1] = float("-inf")   # every token as likely as every other: the first
    want.append(0)
    rows, logits = len(want), logits.cuda()
    got = torch.full((rows,), -7, dtype=torch.int32, device="cuda")
    ops.argmax(logits, got)
    assert got.tolist() == want
    got.fill_(-7)
    zeros = torch.zeros(rows, dtype=torch.int64, device="cuda")
    ops.sample(logits, torch.zeros(rows, device="cuda"), torch.ones(rows, device="cuda"), zeros, zeros, got)
    assert got.tolist() == want
    ops.sample(logits, torch.ones(rows, device="cuda"), torch.full((rows,), 0.9, device="cuda"), zeros, zeros, got)
    assert all(0 <= token < vocab for token in got.tolist()) and got[0].item() == 0


@pytest.mark.parametrize("vocab", [1, 3, 32000, 32767, 32768, 32769, 65537, 128256, 131073, 262145])
def test_sampling_over_blocks_keeps_the_set_and_the_order_of_tokens(ops, vocab):
    """Rows of one block, of clusters of 2 and 4 and of the long kernel, vocabularies at their edges; against sums in 64 bits."""
    torch.manual_seed(35)
    rows = 24
    logits = torch.randn(rows, vocab) * 2
    if vocab > 3:
        logits[:, vocab - 1] = logits[:, vocab // 2] = 9.0   # ties at the top, one of them the last token
        logits[0] = 0.0                                       # every token as probable as every other
    temperature = torch.tensor([0.8, 1.3, 0.0])[torch.arange(rows) % 3]
    top_p = torch.tensor([0.95, 0.5, 1.0, 1e-6])[torch.arange(rows) % 4]
    seeds, counters = torch.arange(rows, dtype=torch.int64) * 3 + 5, torch.arange(rows, dtype=torch.int64)
    got = torch.full((rows,), -7, dtype=torch.int32, device="cuda")
    ops.sample(logits.cuda(), temperature.cuda(), top_p.cuda(), seeds.cuda(), counters.cuda(), got)
    for r, token in enumerate(got.tolist()):
        if float(temperature[r]) == 0.0:
            assert token == int((logits[r] == logits[r].max()).nonzero()[0]), r
            continue
        p = torch.exp((logits[r] - logits[r].max()).double() / float(temperature[r]))
        order = p.sort(descending=True).values
        sums = order.cumsum(0)
        # 32-bit sums: a run of up to 257 terms in order, 1,024 runs in order for the places, each rounding at most 2^-24 of the sum so far
        slack = (257 + 1024) * 2.0 ** -24 * float(sums[-1])
        crossing = min(int((sums < float(top_p[r]) * sums[-1] - slack).sum()), vocab - 1)
        last = min(int((sums < float(top_p[r]) * sums[-1] + slack).sum()), vocab - 1)
        # the threshold is the probability of the token that crosses the line; rounding may move the line by the slack
        assert float(p[token]) >= float(order[last]) * (1 - 1e-5), (r, token)
        if float(top_p[r]) == 1.0 or float(order[crossing]) == float(order[last]):
            kept = torch.where(p >= float(order[crossing]) * (1 - 1e-6) if float(top_p[r]) < 1.0 else p > 0, p, 0.0).cumsum(0)
            target = ops.uniform_from(int(seeds[r]), int(counters[r])) * float(kept[-1])
            before = float(kept[token]) - float(p[token])
            assert before - slack <= target <= float(kept[token]) + slack, (r, token)


@pytest.mark.parametrize("vocab", [3073, 20000, 32768, 40001, 65536, 100000, 131069])
def test_sampling_kernels_draw_what_the_simple_one_draws(ops, vocab):
    """More rows than clusters run at once, greedy ones among them, flat tails (where another order of sums shows) and peaked rows: every draw as the simple kernel's, which
    works with one block and one order of sums at any length."""
    torch.manual_seed(44)
    rows = 161
    logits = (torch.randn(rows, vocab) * torch.tensor([0.3, 1.0, 3.0])[torch.arange(rows) % 3, None]).cuda()
    logits[7], logits[8] = float("nan"), 0.0
    temperature = torch.tensor([0.8, 1.3, 0.0, 0.5, 1.0])[torch.arange(rows) % 5].cuda()
    top_p = torch.tensor([0.95, 0.5, 1.0, 0.999])[torch.arange(rows) % 4].cuda()
    counters = torch.arange(rows, dtype=torch.int64, device="cuda")
    for seed in range(3):
        got, want = (torch.full((rows,), -7, dtype=torch.int32, device="cuda") for _ in range(2))
        seeds = torch.full((rows,), seed, dtype=torch.int64, device="cuda")
        ops.sample(logits, temperature, top_p, seeds, counters, got)
        pointer = lambda t: ops.c_void_p(t.data_ptr())  # noqa: E731
        assert ops.core().tlie_sample_simple(pointer(logits), ops.c_int(rows), ops.c_int(vocab), pointer(temperature), pointer(top_p), pointer(seeds), pointer(counters),
                                             pointer(want), ops._stream()) == 0
        assert torch.equal(got, want)
        assert int(got.min()) >= 0 and int(got.max()) < vocab


def test_argmax_and_sampling(ops):
    torch.manual_seed(7)
    logits = torch.randn(6, 1000)
    logits[0, 10] = logits[0, 700] = 9.0     # a tie: the lowest id wins
    logits[1, 999] = 12.0
    out = torch.empty(6, dtype=torch.int32, device="cuda")
    ops.argmax(logits.cuda(), out)
    want = torch.empty(6, dtype=torch.int32)
    plain_ops.argmax(logits, want)
    assert torch.equal(out.cpu(), want) and int(want[0]) == 10 and int(want[1]) == 999
    # rows long enough for several rounds of the 16-byte loads, maxima at a round's edge, at the end, and tied across rounds
    wide = torch.randn(4, 20000)
    wide[0, 4096 * 4 - 1] = 30.0
    wide[1, 19999] = 30.0
    wide[2, 17001] = wide[2, 4099] = 30.0
    wide[3, 0] = 30.0
    out = torch.empty(4, dtype=torch.int32, device="cuda")
    ops.argmax(wide.cuda(), out)
    assert out.cpu().tolist() == [4096 * 4 - 1, 19999, 4099, 0]
    greedy = torch.empty(4, dtype=torch.int32, device="cuda")
    ops.sample(wide.cuda(), torch.zeros(4).cuda(), torch.ones(4).cuda(), torch.zeros(4, dtype=torch.int64).cuda(), torch.zeros(4, dtype=torch.int64).cuda(), greedy)
    assert greedy.cpu().tolist() == [4096 * 4 - 1, 19999, 4099, 0]
    assert ops.uniform_from(11, 5) == plain_ops.uniform_from(11, 5) == pytest.approx(ops.core().tlie_uniform_from(11, 5))
    rows = 64
    logits = torch.randn(rows, 131) * 2
    temperature = torch.tensor([0.0, 0.8, 1.0, 1.5] * (rows // 4))
    top_p = torch.tensor([1.0, 1.0, 0.9, 0.5, 0.3, 1.0, 0.7, 0.95] * (rows // 8))
    seeds = torch.arange(rows, dtype=torch.int64) * 7 + 1
    counters = torch.arange(rows, dtype=torch.int64) % 5
    got = torch.empty(rows, dtype=torch.int32, device="cuda")
    ops.sample(logits.cuda(), temperature.cuda(), top_p.cuda(), seeds.cuda(), counters.cuda(), got)
    want = torch.empty(rows, dtype=torch.int32)
    plain_ops.sample(logits, temperature, top_p, seeds, counters, want)
    # the two sides sum probabilities in different orders: a draw that lands within rounding of a
    # boundary may fall on the neighbouring kept token, so demand near-total agreement, and exact for greedy rows
    agree = (got.cpu() == want)
    assert bool(agree[temperature == 0].all())
    assert int(agree.sum()) >= rows - 2, (got.cpu(), want)
    # the distribution: many draws of one row follow softmax(l / T) restricted by top_p
    row = torch.tensor([2.0, 1.0, 0.5, -1.0, -3.0] + [-20.0] * 45)
    n = 4096
    got = torch.empty(n, dtype=torch.int32, device="cuda")
    ops.sample(row.repeat(n, 1).cuda(), torch.full((n,), 0.7).cuda(), torch.full((n,), 0.8).cuda(), torch.full((n,), 3, dtype=torch.int64).cuda(), torch.arange(n, dtype=torch.int64).cuda(), got)
    p = torch.softmax(row / 0.7, 0)
    keep = p >= p[1]  # 0.8 is reached by the two most probable tokens
    expect = torch.where(keep, p, torch.zeros_like(p)) / p[keep].sum()
    freq = torch.bincount(got.cpu().long(), minlength=50).float() / n
    assert float((freq - expect).abs().max()) < 0.03


@pytest.mark.parametrize("q_heads,kv_heads,head_dim,page_size", [(8, 1, 64, 64), (4, 4, 64, 16), (6, 2, 128, 32), (24, 2, 64, 16), (32, 1, 128, 16)])
def test_paged_attention_f32_over_shared_keys(ops, q_heads, kv_heads, head_dim, page_size):
    """Rows of one request and of several in a tile, lengths around 32 keys, NaN where no row looks; a row has the same bits alone and among others."""
    torch.manual_seed(34)
    rng = np.random.default_rng(34)
    seq_lens, q_lens = [1, 31, 32, 33, 64, 97, 200], [1, 31, 2, 33, 1, 40, 3]
    qkv, pages, positions, token_seq, table = _paged_case(rng, torch.float32, seq_lens, q_lens, kv_heads, head_dim, page_size, q_heads)
    want = torch.empty(len(positions), q_heads * head_dim)
    plain_ops.paged_attention(qkv, pages, positions, token_seq, table, want, q_heads, kv_heads, head_dim, page_size)
    for entry, length in enumerate(seq_lens):
        if length % page_size:
            pages[int(table[entry, length // page_size]), :, :, length % page_size :] = float("nan")
    args = (pages.cuda(), positions.cuda(), token_seq.cuda(), table.cuda())
    got = torch.empty(want.shape, device="cuda")
    ops.paged_attention(qkv.cuda(), *args, got, q_heads, kv_heads, head_dim, page_size)
    assert torch.allclose(got.cpu(), want, atol=4e-6), float((got.cpu() - want).abs().max())

    class Single:
        decode_only = True

    lasts = torch.tensor(np.cumsum(q_lens) - 1)
    alone = torch.empty(len(lasts), want.shape[1], device="cuda")
    ops.paged_attention(qkv[lasts].cuda(), args[0], positions[lasts].cuda(), torch.arange(len(lasts), dtype=torch.int32).cuda(), args[3], alone,
                        q_heads, kv_heads, head_dim, page_size, batch=Single())
    assert torch.equal(alone, got[lasts.cuda()])


@pytest.mark.parametrize("q_heads,kv_heads,head_dim,page_size", [(8, 1, 64, 64), (4, 4, 64, 16), (6, 2, 128, 32), (24, 2, 64, 16), (32, 1, 128, 16), (9, 9, 128, 64)])
@pytest.mark.parametrize("q_lens", [[1, 1, 1, 1, 40, 3], [2] * 9, [33, 1, 1, 1, 1, 32], [5, 5, 5, 70], [1] * 7, [64], None])
def test_paged_attention_f32_over_shared_keys_has_the_bits_of_the_general_kernel(ops, q_heads, kv_heads, head_dim, page_size, q_lens):
    """Described steps, whose tiles are as tall as their requests allow, and one that nobody describes."""
    torch.manual_seed(41)

    class Batch:
        host_q_lens = q_lens

    lens = q_lens or [3, 30, 1]
    held = [q + (i * 37) % 90 for i, q in enumerate(lens)]
    qkv, pages, positions, token_seq, table = _paged_case(np.random.default_rng(41), torch.float32, held, lens, kv_heads, head_dim, page_size, q_heads)
    qkv, pages, positions, token_seq, table = (t.cuda() for t in (qkv, pages, positions, token_seq, table))
    got, want = (torch.full((len(positions), q_heads * head_dim), float("nan"), device="cuda") for _ in range(2))
    ops.paged_attention(qkv, pages, positions, token_seq, table, got, q_heads, kv_heads, head_dim, page_size, batch=Batch())
    c_int, pointer = ops.c_int, lambda t: ops.c_void_p(t.data_ptr())  # noqa: E731
    status = ops.core().tlie_paged_attention_generic(
        c_int(0), pointer(qkv), c_int(qkv.shape[1]), pointer(pages), pointer(positions), pointer(token_seq), pointer(table), c_int(table.shape[1]), pointer(want),
        c_int(len(positions)), c_int(q_heads), c_int(kv_heads), c_int(head_dim), c_int(page_size), c_int(0), ops.c_float(head_dim ** -0.5), ops._stream())
    assert status == 0
    assert torch.equal(got, want)


@pytest.mark.parametrize("q_heads,kv_heads,head_dim,page_size,window", [
    (32, 4, 64, 64, 0), (8, 8, 128, 64, 0), (32, 8, 128, 16, 0), (4, 2, 16, 16, 0), (6, 2, 32, 32, 0), (3, 3, 48, 16, 0),
    (16, 1, 64, 64, 0), (8, 2, 64, 32, 100), (10, 2, 80, 16, 33),
])
@pytest.mark.parametrize("splits", [1, 3, 16])
def test_decode_attention_split_kv(ops, q_heads, kv_heads, head_dim, page_size, window, splits):
    """The tensor-core decode kernel against the plain function: lengths at page and tile edges, one far key that dominates."""
    from tinyllama_inference_engine_b200.ops import fast

    rng = np.random.default_rng(8)
    torch.manual_seed(8)
    seq_lens = [1, 31, 32, 33, 64, 65, 127, 129, 700, 1153, 2 * page_size, 2 * page_size + 1]
    qkv, pages, positions, token_seq, table = _paged_case(rng, torch.bfloat16, seq_lens, [1] * len(seq_lens), kv_heads, head_dim, page_size, q_heads)
    for row in (8, 9):  # key 3 of the long requests matches every head's query strongly (only visible without a window)
        page, slot = int(table[row, 3 // page_size]), 3 % page_size
        for h in range(q_heads):
            qv = qkv.view(qkv.shape[0], -1, head_dim)[row, h].float()
            pages[page, 0, h // (q_heads // kv_heads), slot] = (qv * (6.0 * head_dim ** 0.5 / float(qv.norm()) ** 2)).bfloat16()
    want = torch.empty(len(seq_lens), q_heads * head_dim, dtype=torch.bfloat16)
    plain_ops.paged_attention(qkv, pages, positions, token_seq, table, want, q_heads, kv_heads, head_dim, page_size, window)
    got = torch.empty(len(seq_lens), q_heads * head_dim, dtype=torch.bfloat16, device="cuda")
    pages_gpu = pages.cuda()
    held = set(int(p) for p in table.flatten() if p >= 0)
    for page in range(pages.shape[0]):   # pages no request holds, and slots past a request's end: reading them would show
        if page not in held:
            pages_gpu[page] = float("nan")
    for i, n in enumerate(seq_lens):
        if n % page_size:
            pages_gpu[int(table[i, n // page_size]), :, :, n % page_size :] = float("nan")
    fast.decode_attention(qkv.cuda(), pages_gpu, positions.cuda(), table.cuda(), got, q_heads, kv_heads, head_dim, page_size, window, head_dim ** -0.5, splits)
    error = (got.cpu().float() - want.float()).abs().max(1).values
    assert float(error.max()) <= 1.6e-2 * 2, error


@pytest.mark.parametrize("q_heads,kv_heads,head_dim,page_size,window", [
    (32, 4, 64, 64, 0), (8, 8, 128, 64, 0), (4, 2, 16, 16, 0), (6, 2, 32, 32, 0), (3, 3, 48, 16, 0), (8, 2, 64, 32, 100), (10, 2, 80, 16, 33), (4, 1, 96, 16, 70),
])
def test_prefill_attention_flash(ops, q_heads, kv_heads, head_dim, page_size, window):
    """The tensor-core prompt kernel against the plain function: portions that start anywhere, tile and page edges, single rows."""
    from tinyllama_inference_engine_b200.ops import fast

    rng = np.random.default_rng(9)
    torch.manual_seed(9)
    seq_lens = [300, 64, 65, 1, 127, 131, 700, 2, 129]
    q_lens = [300, 64, 2, 1, 1, 131, 70, 2, 65]
    qkv, pages, positions, token_seq, table = _paged_case(rng, torch.bfloat16, seq_lens, q_lens, kv_heads, head_dim, page_size, q_heads)
    row = sum(q_lens[:6]) + 69  # the last row of the request of 700: key 5 far behind it dominates (if no window hides it)
    page, slot = int(table[6, 5 // page_size]), 5 % page_size
    for h in range(q_heads):
        qv = qkv.view(qkv.shape[0], -1, head_dim)[row, h].float()
        pages[page, 0, h // (q_heads // kv_heads), slot] = (qv * (6.0 * head_dim ** 0.5 / float(qv.norm()) ** 2)).bfloat16()
    tokens = qkv.shape[0]
    want = torch.empty(tokens, q_heads * head_dim, dtype=torch.bfloat16)
    plain_ops.paged_attention(qkv, pages, positions, token_seq, table, want, q_heads, kv_heads, head_dim, page_size, window)
    starts = np.concatenate([[0], np.cumsum(q_lens)]).astype(np.int32)
    firsts = np.array([s - q for s, q in zip(seq_lens, q_lens)], dtype=np.int32)
    from tinyllama_inference_engine_b200.ops.fast import ATTENTION_TILE_ROWS
    tiles = [[i, int(starts[i]) + off] for i, q in enumerate(q_lens) for off in range(0, q, ATTENTION_TILE_ROWS)]
    pages_gpu = pages.cuda()
    held = set(int(p) for p in table.flatten() if p >= 0)
    for page in range(pages.shape[0]):
        if page not in held:
            pages_gpu[page] = float("nan")
    for i, n in enumerate(seq_lens):
        if n % page_size:
            pages_gpu[int(table[i, n // page_size]), :, :, n % page_size :] = float("nan")
    got = torch.full((tokens, q_heads * head_dim), float("nan"), dtype=torch.bfloat16, device="cuda")
    fast.prefill_attention(qkv.cuda(), pages_gpu, torch.tensor(tiles, dtype=torch.int32).cuda(), torch.from_numpy(starts).cuda(), torch.from_numpy(firsts).cuda(),
                           table.cuda(), got, q_heads, kv_heads, head_dim, page_size, window, head_dim ** -0.5)
    error = (got.cpu().float() - want.float()).abs().max(1).values
    assert float(error.max()) <= 1.6e-2 * 2, (int(error.argmax()), error.max())


@pytest.mark.parametrize("M", [1, 5, 8, 9, 16])
@pytest.mark.parametrize("N,K", [(130, 80), (2560, 2048), (2048, 5632), (1000, 200), (352, 176)])
def test_gemv_fused(ops, M, N, K):
    """The fused decode products: plain, with the norm in front, accumulating into the residual, and gated."""
    from tinyllama_inference_engine_b200.ops import fast

    torch.manual_seed(11)
    x = torch.randn(M, K).bfloat16()
    w = (torch.randn(N, K) * 0.05).bfloat16()
    want = x.float() @ w.float().T
    scale = float(want.abs().max())
    for dtype, tol in ((torch.float32, 1e-4), (torch.bfloat16, 1.6e-2)):
        got = torch.full((M, N), float("nan"), dtype=dtype, device="cuda")
        fast.gemv_fused(x.cuda(), w.cuda(), got)
        assert torch.allclose(got.cpu().float(), want, atol=tol * scale, rtol=0)
    residual = torch.randn(M, N)
    got = residual.clone().cuda()
    fast.gemv_fused(x.cuda(), w.cuda(), got, epilogue="accumulate")
    assert torch.allclose(got.cpu(), residual + want, atol=1e-4 * scale + 1e-5)
    # long rows and few tiles take sixteen warps per CTA (K split sixteen ways): the same sums with the eight-warp kernel
    library = fast.gemv_library()
    library.tlie_gemv_set_wide_ctas(0)
    try:
        narrow = residual.clone().cuda()
        fast.gemv_fused(x.cuda(), w.cuda(), narrow, epilogue="accumulate")
    finally:
        library.tlie_gemv_set_wide_ctas(1)
    assert torch.allclose(narrow, got, atol=1e-4 * scale + 1e-5)
    # gated: silu of the first half of the rows times the second half, both rounded to bfloat16 first
    half = N // 2
    g, u = want[:, :half].bfloat16().float(), want[:, half:].bfloat16().float()
    gated = torch.empty(M, half, dtype=torch.bfloat16, device="cuda")
    fast.gemv_fused(x.cuda(), w.cuda(), gated, epilogue="gated")
    expect = (g / (1 + torch.exp(-g))) * u
    assert torch.allclose(gated.cpu().float(), expect, atol=1.6e-2 * float(expect.abs().max()) + 2e-3 * scale)
    # norm in front, with and without a gather of rows
    stream = torch.randn(M + 3, K) * 2
    norm_weight = 1 + 0.1 * torch.randn(K)
    for rows in (None, torch.randperm(M + 3)[:M].to(torch.int32)):
        normed = torch.empty(M, K, dtype=torch.bfloat16)
        plain_ops.add_rmsnorm(stream.clone(), None, norm_weight, 1e-5, normed, rows if rows is not None else torch.arange(M, dtype=torch.int32))
        want_n = normed.float() @ w.float().T
        got = torch.empty(M, N, dtype=torch.float32, device="cuda")
        fast.gemv_fused(stream.cuda(), w.cuda(), got, norm=(norm_weight.cuda(), 1e-5, None if rows is None else rows.cuda()))
        # the kernel rounds residual * weight to bfloat16 and scales the 32-bit sum: the same product, rounded elsewhere
        assert torch.allclose(got.cpu(), want_n, atol=6e-3 * float(want_n.abs().max())), float((got.cpu() - want_n).abs().max())
    # a product that completes the residual prepares the norm that follows: the next product reads what it left
    # (bfloat16(residual * weight) and the rows' sums of squares) and gives what the norm-in-front kernel gives
    if N % 8 == 0:
        residual = torch.randn(M, N) * 2
        next_weight = 1 + 0.1 * torch.randn(N)
        w2 = (torch.randn(40, N) * 0.05).bfloat16()
        total = residual.clone().cuda()
        x_out, squares = fast.prepared_norm_buffers(M, N, "cuda")
        fast.gemv_fused(x.cuda(), w.cuda(), total, epilogue="accumulate", prepare=(next_weight.cuda(), x_out, squares))
        assert torch.allclose(total.cpu(), residual + want, atol=1e-4 * scale + 1e-5)
        assert torch.equal(x_out.cpu(), (total.cpu() * next_weight).bfloat16())
        assert torch.allclose(squares.sum(1).cpu(), (total.cpu() ** 2).sum(1), rtol=1e-5)
        via_prepared = torch.empty(M, 40, dtype=torch.float32, device="cuda")
        fast.gemv_fused(x_out, w2.cuda(), via_prepared, prepared=(squares, 1e-5))
        via_norm = torch.empty(M, 40, dtype=torch.float32, device="cuda")
        fast.gemv_fused(total, w2.cuda(), via_norm, norm=(next_weight.cuda(), 1e-5, None))
        assert torch.allclose(via_prepared, via_norm, rtol=1e-5, atol=1e-6 * float(via_norm.abs().max()))


@pytest.mark.parametrize("M", [1, 17, 33, 64, 100, 127])
@pytest.mark.parametrize("N,K", [(130, 80), (2560, 2048), (2048, 5632), (1000, 200), (4096, 14336), (32000, 2048)])
def test_gemm_skinny(ops, M, N, K):
    """The weight-streaming tensor-core product of 17 to 127 rows against the 32-bit product: every epilogue, K cut over clusters of
    every size (the shapes give 1 to 8 parts), widths and depths that are no multiple of the tile, and the prepared-norm hand-over."""
    from tinyllama_inference_engine_b200.ops import fast

    torch.manual_seed(13)
    x = torch.randn(M, K).bfloat16()
    w = (torch.randn(N, K) * 0.05).bfloat16()
    want = x.float() @ w.float().T
    scale = float(want.abs().max())
    xc, wc = x.cuda(), w.cuda()
    for dtype, tol in ((torch.float32, 1e-4), (torch.bfloat16, 1.6e-2)):
        got = torch.full((M, N), float("nan"), dtype=dtype, device="cuda")
        fast.gemm_skinny(xc, wc, got)
        error = (got.cpu().float() - want).abs()
        assert float(error.max()) <= tol * scale, (dtype, float(error.max()), scale, divmod(int(error.argmax()), N))
    residual = torch.randn(M, N)
    got = residual.clone().cuda()
    fast.gemm_skinny(xc, wc, got, epilogue="accumulate")
    assert torch.allclose(got.cpu(), residual + want, atol=1e-4 * scale + 1e-5)
    again = residual.clone().cuda()
    fast.gemm_skinny(xc, wc, again, epilogue="accumulate")
    assert torch.equal(again, got)   # the parts are added in rank order: the same bits every time
    half = N // 2
    g, u = want[:, :half].bfloat16().float(), want[:, half:2 * half].bfloat16().float()
    gated = torch.full((M, half), float("nan"), dtype=torch.bfloat16, device="cuda")
    fast.gemm_skinny(xc, wc[: 2 * half], gated, epilogue="gated")
    expect = (g / (1 + torch.exp(-g))) * u
    assert torch.allclose(gated.cpu().float(), expect, atol=1.6e-2 * float(expect.abs().max()) + 2e-3 * scale)
    # a product that completes the residual prepares the norm that follows; the next product scales its results by the rows' norms
    if N <= 4096:
        torch.manual_seed(14)
        residual = torch.randn(M, N) * 2
        next_weight = 1 + 0.1 * torch.randn(N)
        w2 = (torch.randn(72, N) * 0.05).bfloat16()
        total = residual.clone().cuda()
        x_out = torch.full((M, N), float("nan"), dtype=torch.bfloat16, device="cuda")
        squares = torch.full((M, fast.skinny_square_runs(M, N, K) + 3), float("nan"), dtype=torch.float32, device="cuda")[:, :-3]   # rows may be strided
        fast.gemm_skinny(xc, wc, total, epilogue="accumulate", prepare=(next_weight.cuda(), x_out, squares))
        assert torch.allclose(total.cpu(), residual + want, atol=1e-4 * scale + 1e-5)
        assert torch.equal(x_out.cpu(), (total.cpu() * next_weight).bfloat16())
        assert torch.allclose(squares.sum(1).cpu(), (total.cpu() ** 2).sum(1), rtol=1e-5)
        if N % 8 == 0:
            normed = torch.empty(M, N, dtype=torch.bfloat16)
            plain_ops.add_rmsnorm(total.cpu().clone(), None, next_weight, 1e-5, normed)
            want_n = normed.float() @ w2.float().T
            via_prepared = torch.full((M, 72), float("nan"), dtype=torch.float32, device="cuda")
            fast.gemm_skinny(x_out, w2.cuda(), via_prepared, prepared=(squares, 1e-5))
            assert torch.allclose(via_prepared.cpu(), want_n, atol=6e-3 * float(want_n.abs().max())), float((via_prepared.cpu() - want_n).abs().max())
            gated_n = torch.full((M, 36), float("nan"), dtype=torch.bfloat16, device="cuda")
            fast.gemm_skinny(x_out, w2.cuda(), gated_n, epilogue="gated", prepared=(squares, 1e-5))
            gn, un = want_n[:, :36].bfloat16().float(), want_n[:, 36:].bfloat16().float()
            expect_n = (gn / (1 + torch.exp(-gn))) * un
            assert torch.allclose(gated_n.cpu().float(), expect_n, atol=2.5e-2 * float(expect_n.abs().max()) + 6e-3 * float(want_n.abs().max()))
    torch.cuda.synchronize()
    assert int(fast.tcgen05_error_flag(got.device)) == 0, "a bounded wait inside the kernel gave up"


@pytest.mark.parametrize("q_heads,kv_heads,head_dim,page_size,window,rotate", [
    (32, 4, 64, 64, 0, True), (8, 8, 128, 64, 0, True), (6, 2, 32, 32, 0, True), (8, 2, 64, 16, 100, True), (4, 2, 64, 16, 0, False), (12, 3, 96, 16, 0, True),
    (24, 2, 64, 16, 0, True),   # groups of twelve: the tile's upper rows are in use, four of them empty
])
@pytest.mark.parametrize("splits", [1, 5])
def test_decode_attention_with_rotation_and_cache_write(ops, q_heads, kv_heads, head_dim, page_size, window, rotate, splits):
    """The decode kernel doing rope_store's work itself: same output, same pages, as rope_store followed by attention."""
    from tinyllama_inference_engine_b200.ops import fast

    rng = np.random.default_rng(12)
    torch.manual_seed(12)
    seq_lens = [1, 32, 33, 64, 65, 700, 1153, 4097, 2 * page_size + 1]
    qkv, pages, positions, token_seq, table = _paged_case(rng, torch.bfloat16, seq_lens, [1] * len(seq_lens), kv_heads, head_dim, page_size, q_heads)
    inv_freq = None
    if rotate:
        exponent = (np.float32(-2.0) * np.arange(head_dim // 2, dtype=np.float32)) / np.float32(head_dim)
        inv_freq = torch.from_numpy(np.power(np.float32(10000.0), exponent, dtype=np.float32))
    for write in (True, False):
        qkv_plain, pages_plain = qkv.clone(), pages.clone()
        want = torch.empty(len(seq_lens), q_heads * head_dim, dtype=torch.bfloat16)
        plain_ops.attention_step(qkv_plain, positions, token_seq, table, inv_freq, head_dim if rotate else 0, pages_plain, want, q_heads, kv_heads, head_dim, page_size, window, None, write)
        pages_gpu = pages.clone().cuda()
        got = torch.empty(len(seq_lens), q_heads * head_dim, dtype=torch.bfloat16, device="cuda")
        fast.decode_attention(qkv.cuda(), pages_gpu, positions.cuda(), table.cuda(), got, q_heads, kv_heads, head_dim, page_size, window, head_dim ** -0.5, splits,
                              fuse_rope=True, inv_freq=None if inv_freq is None else inv_freq.cuda(), write_cache=write)
        assert float((got.cpu().float() - want.float()).abs().max()) <= 3.2e-2
        assert torch.allclose(pages_gpu.cpu().float(), pages_plain.float(), atol=1.6e-2 * 4 + 2e-4)
        if not write:
            assert torch.equal(pages_gpu.cpu(), pages)


@pytest.mark.parametrize("q_heads,kv_heads,head_dim", [(32, 4, 64), (8, 2, 128)])
@pytest.mark.parametrize("splits", [2, 4, 8, 18])
def test_decode_attention_parts_that_are_warps(ops, q_heads, kv_heads, head_dim, splits):
    """Keys around whole tiles and around as many tiles as a CTA has warps: parts in one CTA, in several, and launched parts without keys."""
    from tinyllama_inference_engine_b200.ops import fast

    rng = np.random.default_rng(36)
    torch.manual_seed(36)
    seq_lens = [1, 31, 32, 33, 64, 65, 96, 97, 128, 129, 255, 256, 257, 288, 577]
    qkv, pages, positions, token_seq, table = _paged_case(rng, torch.bfloat16, seq_lens, [1] * len(seq_lens), kv_heads, head_dim, 64, q_heads)
    want = torch.empty(len(seq_lens), q_heads * head_dim, dtype=torch.bfloat16)
    plain_ops.paged_attention(qkv, pages, positions, token_seq, table, want, q_heads, kv_heads, head_dim, 64)
    for _ in range(2):   # the tickets are left as they were found
        got = torch.empty(want.shape, dtype=torch.bfloat16, device="cuda")
        fast.decode_attention(qkv.cuda(), pages.cuda(), positions.cuda(), table.cuda(), got, q_heads, kv_heads, head_dim, 64, 0, head_dim ** -0.5, splits)
        assert float((got.cpu().float() - want.float()).abs().max()) <= 1.6e-2


@pytest.mark.parametrize("q_heads,kv_heads,head_dim", [(32, 4, 64), (16, 8, 64), (8, 2, 128), (16, 2, 32)])
@pytest.mark.parametrize("splits", [18, 32])
def test_decode_attention_parts_that_are_warps_have_the_bits_of_parts_that_are_ctas(ops, q_heads, kv_heads, head_dim, splits):
    """Every request twice: as it is, and behind eight tiles of keys whose weights are exactly 0, which are too many parts for one CTA and are merged by ticket.  (Parts
    that count for nothing leave the others' sums as they are: added in order, and in the tree over lanes a multiple of eight away.)"""
    from tinyllama_inference_engine_b200.ops import fast

    rng = np.random.default_rng(37)
    torch.manual_seed(37)
    lens = [1, 2, 31, 32, 33, 63, 64, 65, 95, 96, 97, 127, 128, 129, 160, 193, 255, 256]
    count, page_size, empty = len(lens), 64, 4   # pages of 64 keys: 256 keys without weight
    seq_lens = lens + [empty * page_size + n for n in lens]
    qkv, pages, positions, token_seq, table = _paged_case(rng, torch.bfloat16, seq_lens, [1] * len(seq_lens), kv_heads, head_dim, page_size, q_heads)
    qkv.view(len(seq_lens), -1, head_dim)[:, :q_heads, 0] = 4.0
    qkv[count:] = qkv[:count]
    pages[:, 0, :, :, 0] = 0.0
    for i, n in enumerate(lens):
        held = -(-n // page_size)
        pages[table[count + i, empty : empty + held].long()] = pages[table[i, :held].long()]
        pages[table[count + i, :empty].long(), 0] = torch.tensor([-4000.0] + [0.0] * (head_dim - 1), dtype=torch.bfloat16)   # scores below -1,400: 2 to their power is 0
    got = torch.full((len(seq_lens), q_heads * head_dim), float("nan"), dtype=torch.bfloat16, device="cuda")
    fast.decode_attention(qkv.cuda(), pages.cuda(), positions.cuda(), table.cuda(), got, q_heads, kv_heads, head_dim, page_size, 0, head_dim ** -0.5, splits)
    assert bool(got.isfinite().all())
    assert torch.equal(got[:count], got[count:])


@pytest.mark.parametrize("M,N,K", [(128, 128, 64), (128, 256, 128), (2048, 2560, 2048), (300, 200, 136), (2048, 2048, 5632), (129, 1000, 2048), (1000, 131, 80),
                                   (4200, 2500, 72)])
@pytest.mark.parametrize("tile_n,pair", [(width, pair) for width in (128, 160, 192, 256) for pair in (False, True)] + [(288, False), (320, False), (288, True), (384, True), (480, True)])   # the wide tiles: two for single SMs, three for pairs
def test_gemm_tcgen05(ops, M, N, K, tile_n, pair):
    """The tcgen05 / TMA / tensor-memory product against a 32-bit product of the same bfloat16 values, tails included (the last
    shape gives every CTA several tiles at every width, the one-accumulator wide tile too)."""
    from tinyllama_inference_engine_b200.ops import fast

    torch.manual_seed(13)
    x = torch.randn(M, K).bfloat16()
    w = (torch.randn(N, K) * 0.05).bfloat16()
    want = x.float() @ w.float().T
    scale = float(want.abs().max())
    for dtype, tol in ((torch.float32, 1e-4), (torch.bfloat16, 1.6e-2)):
        got = torch.full((M, N), float("nan"), dtype=dtype, device="cuda")
        fast.gemm_tcgen05(x.cuda(), w.cuda(), got, tile_n=tile_n, pair=pair)
        torch.cuda.synchronize()
        assert int(fast.tcgen05_error_flag(got.device)) == 0, "a bounded wait inside the kernel gave up"
        error = (got.cpu().float() - want).abs()
        assert float(error.max()) <= tol * scale, (float(error.max()), scale, int(error.argmax()) // N, int(error.argmax()) % N)


@pytest.mark.parametrize("pair,tile_n", [(False, 256), (True, 256), (True, 384), (True, 480)])
@pytest.mark.parametrize("M,N,K", [(128, 128, 64), (2048, 2048, 5632), (300, 200, 136), (1000, 132, 80), (129, 1000, 2048), (2100, 4100, 72)])
def test_gemm_tcgen05_accumulate(ops, M, N, K, pair, tile_n):
    """residual += product in the product's epilogue (bulk tensor reductions, each element once): twice in a row, tails included."""
    from tinyllama_inference_engine_b200.ops import fast

    torch.manual_seed(17)
    x = torch.randn(M, K).bfloat16()
    w = (torch.randn(N, K) * 0.05).bfloat16()
    start = torch.randn(M, N)
    product = x.float() @ w.float().T
    residual = start.clone().cuda()
    guard = torch.full((M + 1, N), 7.0, device="cuda")   # the rows behind the residual must stay as they are
    view = guard[:M]
    view.copy_(residual)
    for times in (1, 2):
        fast.gemm_tcgen05_accumulate(x.cuda(), w.cuda(), view, pair=pair, tile_n=tile_n)
        torch.cuda.synchronize()
        assert int(fast.tcgen05_error_flag(view.device)) == 0, "a bounded wait inside the kernel gave up"
        want = start + times * product
        error = (view.cpu() - want).abs()
        assert float(error.max()) <= 1e-4 * float(want.abs().max()), (times, float(error.max()), int(error.argmax()) // N, int(error.argmax()) % N)
        assert float((guard[M] - 7.0).abs().max()) == 0.0


@pytest.mark.parametrize("pair", [False, True])
@pytest.mark.parametrize("M,inter,K", [(128, 128, 64), (2048, 5632, 2048), (300, 176, 136), (1000, 200, 80)])
def test_gemm_tcgen05_gated(ops, M, inter, K, pair):
    from tinyllama_inference_engine_b200.ops import fast

    torch.manual_seed(14)
    x = torch.randn(M, K).bfloat16()
    w = (torch.randn(2 * inter, K) * 0.05).bfloat16()
    both = (x.float() @ w.float().T).bfloat16().float()
    g, u = both[:, :inter], both[:, inter:]
    want = (g / (1 + torch.exp(-g))) * u
    got = torch.full((M, inter), float("nan"), dtype=torch.bfloat16, device="cuda")
    fast.gemm_tcgen05_gated(x.cuda(), w.cuda(), got, pair=pair)
    torch.cuda.synchronize()
    assert int(fast.tcgen05_error_flag(got.device)) == 0
    assert float((got.cpu().float() - want).abs().max()) <= 1.6e-2 * float(want.abs().max()) + 2e-3 * float(both.abs().max())


@pytest.mark.parametrize("head_dim", [64, 128])
@pytest.mark.parametrize("q_heads,kv_heads,page_size,window", [(32, 4, 64, 0), (8, 2, 64, 100), (4, 4, 128, 0), (16, 1, 64, 37), (3, 3, 64, 0)])
def test_prefill_attention_tensor_memory(ops, q_heads, kv_heads, page_size, window, head_dim):
    """The tcgen05 prompt kernel (head size 64 and 128) against the plain function: portions that start anywhere, page edges, single rows."""
    from tinyllama_inference_engine_b200.ops.fast import paired_attention_tiles
    from tinyllama_inference_engine_b200.ops import fast

    rng = np.random.default_rng(15)
    torch.manual_seed(15)
    seq_lens = [300, 64, 65, 1, 127, 131, 700, 2, 129, 1000]
    q_lens = [300, 64, 2, 1, 1, 131, 70, 2, 65, 512]
    qkv, pages, positions, token_seq, table = _paged_case(rng, torch.bfloat16, seq_lens, q_lens, kv_heads, head_dim, page_size, q_heads)
    row = sum(q_lens[:6]) + 69
    page, slot = int(table[6, 5 // page_size]), 5 % page_size
    for h in range(q_heads):
        qv = qkv.view(qkv.shape[0], -1, head_dim)[row, h].float()
        pages[page, 0, h // (q_heads // kv_heads), slot] = (qv * (6.0 * head_dim ** 0.5 / float(qv.norm()) ** 2)).bfloat16()
    # A score far above everything before it, many key tiles into a row (request 9, position 588, key 568): the kernel keeps its
    # running output in tensor memory against a reference maximum and must rescale it there when the maximum jumps.
    late_row = sum(q_lens[:9]) + 100
    page, slot = int(table[9, 568 // page_size]), 568 % page_size
    for h in range(q_heads):
        qv = qkv.view(qkv.shape[0], -1, head_dim)[late_row, h].float()
        pages[page, 0, h // (q_heads // kv_heads), slot] = (qv * (16.0 * head_dim ** 0.5 / float(qv.norm()) ** 2)).bfloat16()
    tokens = qkv.shape[0]
    want = torch.empty(tokens, q_heads * head_dim, dtype=torch.bfloat16)
    plain_ops.paged_attention(qkv, pages, positions, token_seq, table, want, q_heads, kv_heads, head_dim, page_size, window)
    starts = np.concatenate([[0], np.cumsum(q_lens)]).astype(np.int32)
    firsts = np.array([s - q for s, q in zip(seq_lens, q_lens)], dtype=np.int32)
    tiles = paired_attention_tiles(q_lens, [int(f) for f in firsts], [int(x) for x in starts])
    assert len(tiles) // 4 == (sum(-(-q // 128) for q in q_lens) + 1) // 2
    pages_gpu = pages.cuda()
    held = set(int(p) for p in table.flatten() if p >= 0)
    for page in range(pages.shape[0]):
        if page not in held:
            pages_gpu[page] = float("nan")
    for i, n in enumerate(seq_lens):
        if n % page_size:
            pages_gpu[int(table[i, n // page_size]), :, :, n % page_size :] = float("nan")
    got = torch.full((tokens, q_heads * head_dim), float("nan"), dtype=torch.bfloat16, device="cuda")
    fast.prefill_attention_tc(qkv.cuda(), pages_gpu, torch.tensor(tiles, dtype=torch.int32).view(-1, 4).cuda(), torch.from_numpy(starts).cuda(), torch.from_numpy(firsts).cuda(),
                              table.cuda(), got, q_heads, kv_heads, head_dim, page_size, window, head_dim ** -0.5)
    torch.cuda.synchronize()
    assert int(fast.tcgen05_error_flag(got.device)) == 0, "a bounded wait inside the kernel gave up"
    error = (got.cpu().float() - want.float()).abs().max(1).values
    assert float(error.max()) <= 1.6e-2 * 2, (int(error.argmax()), float(error.max()))


def test_hardware_probes_report_what_the_designs_rest_on():
    """The loops of csrc/probes.cu run to the end (every wait in them is bounded) and say what the kernels assume: a tensor-core
    product of 256 columns takes about twice one of 128, narrower ones cost no less than a floor, and a completed barrier is cheap."""
    from tinyllama_inference_engine_b200.ops.probes import hardware_probes

    report = hardware_probes("cuda:0")
    mma = report["mma_cycles"]
    wide, half, narrow = (mma[f"128 x {n} x 16, straight-line issue, one CTA per SM"] for n in (256, 128, 64))
    assert 100 < wide < 200 and 1.6 < wide / half < 2.4 and narrow <= half + 8
    assert mma["128 x 64 x 16, straight-line issue, two CTAs per SM"] > 1.5 * narrow       # two CTAs share one tensor core
    assert 0 < report["handoff_cycles"]["wait on a completed barrier"] < 400
    alone = report["arithmetic_cycles_per_64_values"]["64 exp2, one warp per scheduler"]
    shared = report["arithmetic_cycles_per_64_values"]["64 exp2, two warps per scheduler"]
    assert 400 < alone < 1200 and shared > 1.4 * alone                                       # the exponential unit is what two warps wait for


def test_product_comparison_runs_every_form(ops):
    """The committed comparison of the engine's products with the library's (kernel-bench --products) runs all forms at a small shape."""
    from tinyllama_inference_engine_b200.ops.probes import product_comparison

    report = product_comparison(256, 256, 512, 384, "cuda:0", launches=3)
    assert set(report) == {"qkv", "o", "gate_up", "down"}
    for line in report.values():
        assert line["own, one SM"] > 0 and line["own, SM pairs"] > 0 and any(key.startswith("library") and value > 0 for key, value in line.items())
        assert line["own_runs"] is False   # 256 rows: the library's


@pytest.mark.parametrize("M", [1, 8, 16])
def test_products_of_very_long_rows_stay_in_the_fused_kernel(ops, M):
    """K = 14,336 (the down projection of the 8B shapes): eight staged rows of x would not fit the kernel's shared memory, but with no
    more tiles than CTA slots nothing is staged at all, so the product and its residual add stay one kernel of this engine."""
    from tinyllama_inference_engine_b200.ops import fast

    torch.manual_seed(13)
    N, K = 4096, 14336
    x = torch.randn(M, K).bfloat16()
    w = (torch.randn(N, K) * 0.02).bfloat16()
    want = x.float() @ w.float().T
    scale = float(want.abs().max())
    residual = torch.randn(M, N)
    assert fast.gemv_fits(M, K, norm=False, N=N) and not fast.gemv_fits(M, K, norm=False)
    before = fast.library_gemm_calls
    got = residual.clone().cuda()
    ops.linear_accumulate(x.cuda(), w.cuda(), got)
    assert torch.allclose(got.cpu(), residual + want, atol=1e-4 * scale + 1e-5)
    out = torch.empty(M, N, dtype=torch.bfloat16, device="cuda")
    ops.linear(x.cuda(), w.cuda(), out)
    assert torch.allclose(out.cpu().float(), want, atol=1.6e-2 * scale, rtol=0)
    assert fast.library_gemm_calls == before
