"""The GEMM that expands packed weights into tensor memory, at the sizes where its split can go wrong, against the CPU checker.

Row counts around the 16-row granularity of the activation block, the switch from two accumulator sets to one (128) and the
largest block (256; beyond 192 rows matrices of long K and few weight rows run this kernel: two activation slots of one slice each);
weight rows that end inside a 16-row tile and inside a 128-row group; one super-block, an odd number, and enough to cut every output
tile over several CTAs (partial sums and arrival counters: a second call must agree bit for bit).  That this kernel ran shows in the
number of launches: the shared-memory GEMM would split K on the shapes beyond 192 rows and add a third.  Weights and activations are rounded to fp16 (2^-11 each, independent), sums are fp32: expected relative L2 error
2e-4 to 4e-4, bar 1e-3."""
import numpy as np
import pytest
import torch

import oracle
import tattletale_b200 as ttq
from conftest import rel_l2
from gpu_util import ALL_FMTS, FMT_IDS, OFMT, make_weight, make_x, odt, x_bits

pytestmark = pytest.mark.gpu
TOL = 1e-3


@pytest.mark.parametrize("fmt", ALL_FMTS, ids=FMT_IDS)
@pytest.mark.parametrize("n,k,m", [(16, 256, 17), (100, 512, 32), (130, 768, 33), (1000, 1024, 48), (256, 2304, 112), (4096, 512, 128),
                                   (264, 1280, 129), (3000, 2560, 144), (130, 8192, 193), (264, 8192, 224), (264, 8192, 241), (264, 8192, 256)])
def test_matches_checker(ctx, fmt, n, k, m):
    dtype = torch.float16 if m % 2 else torch.bfloat16
    blocks = make_weight(fmt, n, k, seed=n + k + m)
    x = make_x(m, k, seed=m + 1, dtype=dtype)
    bias = torch.from_numpy(np.random.default_rng(m).normal(0, 0.1, n).astype(np.float32))
    lin = ttq.QuantLinear(ctx, fmt, torch.from_numpy(blocks), k, bias=bias.cuda())
    xd = x.cuda()
    before = ctx.launch_count
    y = lin.forward(xd, out_dtype=torch.float32)
    assert ctx.launch_count - before == 2
    again = lin.forward(xd, out_dtype=torch.float32)
    ctx.check_device_status()
    want = oracle.linear(OFMT[fmt], blocks, x_bits(x), odt(dtype), bias.numpy())
    assert rel_l2(y.cpu().numpy(), want) < TOL
    assert torch.equal(y, again)
    lin.close()


@pytest.mark.parametrize("fmt", ALL_FMTS, ids=FMT_IDS)
def test_rows_of_a_wider_matrix(ctx, fmt):
    """x and y as column slices of wider tensors: row pitches larger than the row, addresses off the 16-byte grid."""
    n, k, m = 200, 512, 50
    blocks = make_weight(fmt, n, k, seed=5)
    wide = make_x(m, k + 9, seed=6).cuda()
    x = wide[:, 3:3 + k]
    out = torch.zeros(m, n + 5, dtype=torch.bfloat16, device="cuda")
    lin = ttq.QuantLinear(ctx, fmt, torch.from_numpy(blocks), k)
    want = lin.forward(x.contiguous())
    lin.forward(x, out=out[:, :n])
    ctx.check_device_status()
    assert torch.equal(out[:, :n], want) and not out[:, n:].any()
    lin.close()


@pytest.mark.parametrize("t,n_exp,top_k", [(24, 32, 4), (9, 8, 8), (130, 8, 1), (250, 8, 4)])
def test_grouped_row_tiles(ctx, t, n_exp, top_k):
    """The expert layer at 16-, 32- and 128-row tiles: fewer items than CTAs, experts with more rows than a tile, every choice dropped."""
    from test_moe_gpu import build, check, routing

    hidden, inter = 1024, 768
    layer, gu, dn = build(ctx, n_exp, hidden, inter, top_k, max_tokens=256, seed=n_exp + t)
    ids, w = routing(t, n_exp, top_k, seed=t, skew=True)
    got = check(ctx, layer, gu, dn, t, hidden, ids, w, seed=t)
    none = check_dropped(ctx, layer, t, hidden, ids, w)
    assert np.isfinite(got).all() and not none.any()
    layer.close()


def check_dropped(ctx, layer, t, hidden, ids, w):
    y = layer.forward(make_x(t, hidden, 1).cuda(), torch.full(ids.shape, -1, dtype=torch.int32, device="cuda"), torch.from_numpy(w).cuda())
    ctx.check_device_status()
    return y.float().cpu().numpy()


@pytest.mark.parametrize("fmt", [ttq.FMT_Q8_0, ttq.FMT_Q6_K], ids=["q8_0", "q6_k"])
@pytest.mark.parametrize("n,k,m", [(76800, 256, 5), (9500, 2048, 8), (4130, 4608, 6), (2000, 9984, 7)])
def test_exact_form_of_five_to_eight_rows(ctx, fmt, n, k, m):
    """Weights as pairs of fp16 values (remainder below 2^-22 of the weight), activations exact after a power of two: what is left is
    the fp32 accumulation; bar 3e-5, the error of the integer decode kernel's 16-bit fixed point.  A power of two on a row
    multiplies its outputs by exactly that, far outside the range of fp16."""
    dtype = torch.float16 if m % 2 else torch.bfloat16
    blocks = make_weight(fmt, n, k, seed=n + k + m)
    x = make_x(m, k, seed=m + 1, dtype=dtype)
    bias = torch.from_numpy(np.random.default_rng(m).normal(0, 0.1, n).astype(np.float32))
    lin = ttq.QuantLinear(ctx, fmt, torch.from_numpy(blocks), k, bias=bias.cuda())
    y = lin.forward(x.cuda(), out_dtype=torch.float32)
    want = oracle.linear(OFMT[fmt], blocks, x_bits(x), odt(dtype), bias.numpy())
    assert rel_l2(y.cpu().numpy(), want) < 3e-5
    wide = x.to(torch.bfloat16).cuda()
    factor = torch.ones(m, 1, device="cuda")
    factor[0], factor[1], factor[m - 1] = 2.0 ** 60, 2.0 ** -60, 0.0
    plain = lin.forward(wide, out_dtype=torch.float32, use_bias=False)
    scaled = lin.forward((wide * factor).to(torch.bfloat16), out_dtype=torch.float32, use_bias=False)
    ctx.check_device_status()
    assert torch.equal(scaled, plain * factor)
    lin.close()


@pytest.mark.parametrize("fmt", [ttq.FMT_Q8_0, ttq.FMT_Q6_K], ids=["q8_0", "q6_k"])
def test_exact_form_of_rows_up_to_the_largest_bf16_value(ctx, fmt):
    """A row whose largest magnitude is the largest finite bf16 value, 1.9921875 * 2^127: its outputs are those of the same row without
    the power of two, times that power."""
    n, k, m = 9500, 2048, 5
    x = make_x(m, k, seed=9).clamp(-6, 6)
    x[0, 77], x[3, k - 1] = 1.9921875 * 4, -1.9921875 * 4
    factor = torch.ones(m, 1)
    factor[0] = factor[3] = 2.0 ** 125
    lin = ttq.QuantLinear(ctx, fmt, torch.from_numpy(make_weight(fmt, n, k, seed=8)), k)
    plain = lin.forward(x.cuda(), out_dtype=torch.float32)
    scaled = lin.forward((x * factor).to(torch.bfloat16).cuda(), out_dtype=torch.float32)
    ctx.check_device_status()
    assert plain.abs().max() < 8 and torch.equal(scaled, plain * factor.cuda())
    lin.close()


@pytest.mark.parametrize("top", [300.0, 1.0e4, 6.0e4])
@pytest.mark.parametrize("fmt", [ttq.FMT_Q8_0, ttq.FMT_Q6_K], ids=["q8_0", "q6_k"])
def test_exact_form_of_weights_beyond_fp16(ctx, fmt, top):
    """Block scales up to `top`, so that weights leave fp16 (at 6e4 Q6_K weights reach 2^27), beside blocks of ordinary scale in the same
    rows and in rows of their own (every third).  The weights of a row are divided by a power of two that keeps its largest below 2^15:
    what is left out is below 2^-32 of that, so the bar of the exact form (3e-5) stands for both kinds of rows."""
    n, k, m = 9500, 2048, 6
    blocks = make_weight(fmt, n, k, seed=31)
    off, size = (0, 34) if fmt == ttq.FMT_Q8_0 else (208, 210)
    b = blocks.reshape(n, -1, size)
    d = np.ascontiguousarray(b[..., off:off + 2]).view(np.float16)[..., 0].astype(np.float64)
    factor = np.where(np.random.default_rng(32).random(d.shape) < 0.5, top / np.abs(d).max(), 1.0)
    factor[::3] = 1.0
    b[..., off:off + 2] = (d * factor).astype(np.float16)[..., None].view(np.uint8).reshape(*d.shape, 2)
    x = make_x(m, k, seed=33)
    lin = ttq.QuantLinear(ctx, fmt, torch.from_numpy(blocks), k)
    on_device = ttq.QuantLinear(ctx, fmt, torch.from_numpy(blocks).cuda(), k)
    y = lin.forward(x.cuda(), out_dtype=torch.float32)
    same = on_device.forward(x.cuda(), out_dtype=torch.float32)
    ctx.check_device_status()
    want = oracle.linear(OFMT[fmt], blocks, x_bits(x), odt(torch.bfloat16), None)
    got = y.cpu().numpy()
    assert np.isfinite(got).all() and torch.equal(y, same)
    assert rel_l2(got, want) < 3e-5
    assert rel_l2(got[:, ::3], want[:, ::3]) < 3e-5
    lin.close()
    on_device.close()


def run_on_two_streams(ctx, first, second, rounds=20):
    """Both calls' results in turn, then enqueued side by side: every round must give the same bits."""
    want = first().clone(), second().clone()
    streams = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    for _ in range(rounds):
        got = []
        for stream, call in zip(streams, (first, second)):
            with torch.cuda.stream(stream):
                got.append([call() for _ in range(4)])
        torch.cuda.synchronize()
        assert all(torch.equal(y, w) for ys, w in zip(got, want) for y in ys)
    ctx.check_device_status()


@pytest.mark.parametrize("beside", ["linear", "layer"])
def test_expert_layer_beside_another_call(ctx, beside):
    """An expert layer keeps its partial sums and arrival counters to itself: a linear of the same context or a second layer may run
    on another stream at the same time."""
    from test_moe_gpu import build, routing

    hidden, inter, n_exp, top_k, t = 1024, 768, 32, 4, 24
    ids, w = (torch.from_numpy(v).cuda() for v in routing(t, n_exp, top_k, seed=3))
    x = make_x(t, hidden, 5).cuda()
    layer = build(ctx, n_exp, hidden, inter, top_k, max_tokens=64, seed=41)[0]
    if beside == "layer":
        other = build(ctx, n_exp, hidden, inter, top_k, max_tokens=64, seed=42)[0]
        call = lambda: other.forward(x, ids, w)
    else:
        other = ttq.QuantLinear(ctx, ttq.FMT_Q4_K, torch.from_numpy(make_weight(ttq.FMT_Q4_K, 2048, 4096, seed=43)), 4096)
        rows = make_x(64, 4096, 6).cuda()
        call = lambda: other.forward(rows)
    run_on_two_streams(ctx, lambda: layer.forward(x, ids, w), call)
    layer.close()
    other.close()


def test_prefill_rows_beside_decode_rows(ctx):
    """Q4_K at 64 rows (the tensor-memory kernel) and at 8 rows of a long K (the one-launch kernel, K cut over CTAs) on two streams: each
    counts the arrivals of its pieces on counters of its own."""
    big = ttq.QuantLinear(ctx, ttq.FMT_Q4_K, torch.from_numpy(make_weight(ttq.FMT_Q4_K, 2048, 4096, seed=51)), 4096)
    long = ttq.QuantLinear(ctx, ttq.FMT_Q4_K, torch.from_numpy(make_weight(ttq.FMT_Q4_K, 1024, 14336, seed=52)), 14336)
    x64, x8 = make_x(64, 4096, 53).cuda(), make_x(8, 14336, 54).cuda()
    run_on_two_streams(ctx, lambda: big.forward(x64), lambda: long.forward(x8))
    big.close()
    long.close()


def test_exact_rows_of_a_host_batch_beside_a_prefill(ctx):
    """Q8_0 at six rows in a recorded batch, which runs on the context's own stream, while a 64-row linear is in flight on the caller's: the
    exact form has its own images, partial sums and counters."""
    n, k = 9500, 2048
    small = ttq.QuantLinear(ctx, ttq.FMT_Q8_0, torch.from_numpy(make_weight(ttq.FMT_Q8_0, n, k, seed=61)), k)
    big = ttq.QuantLinear(ctx, ttq.FMT_Q4_K, torch.from_numpy(make_weight(ttq.FMT_Q4_K, 4096, 4096, seed=62)), 4096)
    x6, x64 = make_x(6, k, 63).pin_memory(), make_x(64, 4096, 64).cuda()
    y6 = torch.zeros(6, n, dtype=torch.bfloat16).pin_memory()
    batch = ttq.HostBatch(ctx, [(small, x6, y6)])
    batch.run()
    want6, want64 = y6.clone(), big.forward(x64)
    torch.cuda.synchronize()
    for _ in range(20):
        y6.zero_()
        ys = [big.forward(x64) for _ in range(8)]
        batch.run()
        torch.cuda.synchronize()
        assert torch.equal(y6, want6) and all(torch.equal(y, want64) for y in ys)
    ctx.check_device_status()
    batch.close()
    small.close()
    big.close()


@pytest.mark.parametrize("t,n_exp,top_k", [(250, 8, 4), (600, 64, 8), (1100, 16, 1)])
def test_expert_layer_repeats_itself(ctx, t, n_exp, top_k):
    """Experts with more rows than a tile: a row lies in the same tile in every call, so its sum has the same order and the same bits."""
    from test_moe_gpu import build, routing

    hidden, inter = 1024, 768
    layer = build(ctx, n_exp, hidden, inter, top_k, max_tokens=t, seed=71)[0]
    ids, w = (torch.from_numpy(v).cuda() for v in routing(t, n_exp, top_k, seed=72, skew=True))
    ids[5, 0] = -1
    x = make_x(t, hidden, 73).cuda()
    first = layer.forward(x, ids, w, out=torch.empty(t, hidden, device="cuda"))
    for _ in range(20):
        assert torch.equal(layer.forward(x, ids, w, out=torch.empty(t, hidden, device="cuda")), first)
    ctx.check_device_status()
    layer.close()
