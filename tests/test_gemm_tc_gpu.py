"""The prompt-sized W4A16 product (more than 16 rows: tcgen05 / tensor-memory kernel behind qb_marlin_gemm) against
the CPU oracle and against the skinny kernel run in 16-row slabs on the same buffers."""
import numpy as np
import pytest
import torch

from oracle import ref_ops as R
from qwenny_b200 import host, synth

pytestmark = pytest.mark.gpu
RTOL, ATOL = 1e-2, 2e-3  # the benchmark's tolerance for product outputs, after rounding to bf16


def bf16(a):
    return torch.as_tensor(np.asarray(a, dtype=np.float32)).to(torch.bfloat16).float().numpy()


def close(a, b):
    a, b = bf16(a), bf16(b)
    return np.abs(a - b) <= ATOL + RTOL * np.abs(b)


def make(rows, cols, silu, seed, m):
    g = synth.gen(seed)
    x = synth.activations(m, cols, g)
    codes, sc = synth.int4_matrix(rows, cols, g)
    words, s16 = host.pack_marlin(codes, sc, silu=silu)
    wdq = R.dequant(codes, sc.astype(np.float16))[R.row_order(rows, silu)]
    dev = lambda a: torch.from_numpy(a).cuda()
    return x, wdq, dev(x), dev(words.view(np.int32)), dev(s16.view(np.int16)).view(torch.float16)


@pytest.mark.parametrize("m,rows,cols", [(64, 256, 128), (256, 512, 1024), (300, 512, 640), (17, 256, 256),
                                         (2048, 1024, 5120)])
def test_plain_vs_oracle_and_slabs(ctx, m, rows, cols):
    x, wdq, xd, wd, sd = make(rows, cols, False, 100 + m, m)
    y = ctx.marlin_gemm(xd, wd, sd)
    torch.cuda.synchronize()
    assert ctx.device_error() == 0
    want = R.marlin_gemm(x, wdq)
    a = y.cpu().numpy()
    assert close(a, want).all()
    # f32 sums of the same f16 products as the oracle's f64: far inside the tolerance
    assert np.abs(a - want).max() < 2e-4 * max(1.0, np.abs(want).max())
    ctx.tune(nstages=-1)  # the skinny kernel in 16-row slabs
    try:
        ys = ctx.marlin_gemm(xd, wd, sd).cpu().numpy()
    finally:
        ctx.tune()
    assert np.abs(a - ys).max() < 2e-4 * max(1.0, np.abs(want).max())


@pytest.mark.parametrize("m,rows,cols", [(128, 512, 256), (2048, 1024, 1024)])
def test_silu_vs_oracle(ctx, m, rows, cols):
    x, wdq, xd, wd, sd = make(rows, cols, True, 200 + m, m)
    y = ctx.marlin_gemm(xd, wd, sd, epi="silu")
    torch.cuda.synchronize()
    assert ctx.device_error() == 0
    want = R.marlin_gemm(x, wdq, "silu")
    assert y.shape == (m, rows // 2)
    assert close(y.float().cpu().numpy(), want.astype(np.float32)).all()


def test_row0_and_prefill_chunk_shape(ctx):
    """Rows row0 .. of a larger X / Y, and the 27B in-projection's width at a 2048-row chunk (sampled columns)."""
    x, wdq, xd, wd, sd = make(512, 384, False, 321, 100)
    y = torch.zeros(100, 512, device="cuda")
    ctx.marlin_gemm(xd, wd, sd, y=y, row0=30, m=50)
    want = R.marlin_gemm(x[30:80], wdq)
    a = y.cpu().numpy()
    assert close(a[30:80], want).all() and np.all(a[:30] == 0) and np.all(a[80:] == 0)


@pytest.mark.parametrize("m,rows,cols,silu", [(600, 1024, 2048, False), (2048, 5120, 1024, False), (520, 512, 1536, True)])
def test_shares_of_the_tile_list_repeat_and_agree_with_whole_tiles(ctx, m, rows, cols, silu):
    """The product deals (tile, k block) pairs to a persistent grid in equal contiguous shares when there are few tiles
    per SM; tiles cut between blocks are summed in block order by the tile's last arriver, so a repeated launch gives
    the same bits, and the result agrees with the same launch run as whole tiles (only the order of the f32 sums over
    k differs) and with the oracle."""
    x, wdq, xd, wd, sd = make(rows, cols, silu, 400 + m, m)
    epi = "silu" if silu else "plain"
    ctx.tune(ctas=1000)  # equal shares whatever the shape
    try:
        a = ctx.marlin_gemm(xd, wd, sd, epi=epi)
        b = ctx.marlin_gemm(xd, wd, sd, epi=epi)
        ctx.tune(ctas=1001)  # whole tiles whatever the shape
        c = ctx.marlin_gemm(xd, wd, sd, epi=epi)
    finally:
        ctx.tune()
    torch.cuda.synchronize()
    assert ctx.device_error() == 0
    assert torch.equal(a, b)
    want = R.marlin_gemm(x, wdq, epi)
    an, cn = a.float().cpu().numpy(), c.float().cpu().numpy()
    assert close(an, want.astype(np.float32)).all() and close(cn, want.astype(np.float32)).all()
    assert np.abs(an - cn).max() <= (2e-3 if silu else 2e-4) * max(1.0, np.abs(want).max())


@pytest.mark.parametrize("m,rows,cols,silu", [(65, 256, 4096, False), (70, 512, 6144, True), (100, 5120, 2048, False), (256, 1280, 5248, False),
                                               (300, 9728, 256, True)])
def test_tiles_cut_into_parts_and_unaligned_results(ctx, m, rows, cols, silu):
    """Few tiles with a long k are cut into parts (down to a stage of 128 per pair of blocks; 5248 columns are 41 stages, which no number
    of pairs divides), many more tiles than pairs are dealt in rounds: the oracle's values and the same bits in a repeated launch. A result that starts off a
    16-byte boundary takes plain stores: the same bits, and nothing beside it is written. Only the order of the f32 sums over k may differ
    from whole tiles: 2e-4 of the largest value (2e-3 where the result is f16), as above."""
    x, wdq, xd, wd, sd = make(rows, cols, silu, 500 + m, m)
    epi, n, dt = ("silu", rows // 2, torch.float16) if silu else ("plain", rows, torch.float32)
    a = ctx.marlin_gemm(xd, wd, sd, epi=epi)
    b = ctx.marlin_gemm(xd, wd, sd, epi=epi)
    room = torch.full((m * n + 9,), 7.0, dtype=dt, device="cuda")
    ctx.marlin_gemm(xd, wd, sd, epi=epi, y=room[1:])
    try:
        ctx.tune(ctas=1001)
        c = ctx.marlin_gemm(xd, wd, sd, epi=epi)
    finally:
        ctx.tune()
    torch.cuda.synchronize()
    assert ctx.device_error() == 0
    assert torch.equal(a, b) and torch.equal(room[1:1 + m * n].view(m, n), a)
    assert room[0] == 7 and (room[1 + m * n:] == 7).all()
    want = R.marlin_gemm(x, wdq, epi)
    an, cn = a.float().cpu().numpy(), c.float().cpu().numpy()
    assert close(an, want.astype(np.float32)).all()
    assert np.abs(an - cn).max() <= (2e-3 if silu else 2e-4) * max(1.0, np.abs(want).max())


@pytest.mark.parametrize("m,rows,cols,zp", [(70, 1024, 1024, False), (100, 256, 17408, False), (256, 2048, 2048, False), (1565, 2048, 2048, False),
                                             (2048, 2048, 2048, False), (700, 5120, 6144, False), (1000, 5120, 17408, False), (333, 5120, 6144, True)])
def test_no_accumulator_runs_longer_than_shares_or_its_tile(ctx, m, rows, cols, zp):
    """The tensor core cuts its f32 sums off: an accumulator loses 1.5e-7 of the result per stage of 128 columns (measured over 1 to 136 of
    them), and joining the parts in f32 some 1e-7. So the error against 64 bits tells the longest part: a tile's whole k only where whole tiles
    fill five sixths of the pairs' rounds, an equal share of all stages elsewhere, with and without zero points."""
    g = synth.gen(700 + m)
    pairs = torch.cuda.get_device_properties(0).multi_processor_count // 2
    tiles, k = rows // 256 * -(-m // 256), cols // 128
    longest = k if 6 * tiles > 5 * -(-tiles // pairs) * pairs else min(k, -(-tiles * k // pairs))
    codes, sc = synth.int4_matrix(rows, cols, g)
    zeros = torch.randint(0, 16, (rows, cols // 128), generator=g, dtype=torch.uint8).numpy() if zp else None
    words, s16 = host.pack_marlin(codes, sc, zeros=zeros)
    xd = torch.from_numpy(synth.activations(m, cols, g)).cuda()
    y = ctx.marlin_gemm(xd, torch.from_numpy(words.view(np.int32)).cuda(), torch.from_numpy(s16.view(np.int16)).cuda().view(torch.float16), zp=zp)
    s = sc.astype(np.float16)
    wdq = R.dequant_z(codes, s, ((8.0 - zeros.astype(np.float32)) * sc).astype(np.float16)) if zp else R.dequant(codes, s)
    wdq = torch.from_numpy(wdq[R.row_order(rows, False)]).cuda().double()  # (as rounded to f16: the sums' error is all there is)
    want = xd.double() @ wdq.T
    err = float((y.double() - want).norm() / want.norm())
    assert err < 1e-7 + 1.7e-7 * longest, (err, longest)
    assert ctx.device_error() == 0


@pytest.mark.parametrize("m,rows,cols", [(17, 256, 128), (32, 512, 384), (33, 256, 640), (40, 1024, 2048), (63, 768, 256),
                                         (64, 2048, 1152), (70, 512, 512), (130, 256, 256)])
def test_few_rows_gathered_argmax_vs_oracle(ctx, m, rows, cols):
    """17 .. 64 rows (and slabs of 64 beyond): edges of the token tile, one group of k and many, gathered rows in any order
    with repeats, the greedy key over part of the outputs. The sums are f32 of exact products, scaled once per group of
    128: an error of at most k / 16 roundings of partial sums, far below 1e-5 of the largest result here."""
    x, wdq, xd, wd, sd = make(rows, cols, False, 500 + m, m + 5)
    order = np.random.default_rng(m).integers(0, m + 5, m).astype(np.int32)
    valid = rows - 100
    keys = torch.zeros(m, dtype=torch.int64, device="cuda")
    y = ctx.marlin_gemm(xd, wd, sd, epi="argmax", xrows=torch.from_numpy(order).cuda(), keys=keys, n_valid=valid)
    torch.cuda.synchronize()
    assert ctx.device_error() == 0
    want = R.marlin_gemm(x[order], wdq)
    a = y.cpu().numpy()
    assert np.abs(a - want).max() < 1e-5 * np.abs(want).max()
    assert (keys.cpu().numpy().view(np.uint64) == R.argmax_keys(a, valid)).all()
    again = torch.zeros_like(keys)
    assert torch.equal(y, ctx.marlin_gemm(xd, wd, sd, epi="argmax", xrows=torch.from_numpy(order).cuda(), keys=again, n_valid=valid))
    assert torch.equal(keys, again)


@pytest.mark.parametrize("m,rows,cols", [(17, 16384, 5120), (40, 65536, 5120), (64, 34816, 5120), (70, 16384, 5120), (48, 5120, 17408)])
def test_few_rows_over_long_shares(ctx, m, rows, cols):
    """The layer's sizes and an output layer, where a block walks tens of stages (the rings and accumulators turn over many times)
    through the tail of one tile, whole tiles and the head of another: sampled outputs against the exact product (the
    bound of the test above), the greedy keys of all outputs, the same bits on repeat, and contiguous rows with the bits
    of the same rows gathered, plain and SwiGLU."""
    from qwenny_b200 import model as M
    g = torch.Generator(device="cuda").manual_seed(800 + m)
    w, x = M.Marlin.random(rows, cols, g), torch.randn(m + 5, cols, generator=g, device="cuda").half()
    order = torch.randint(0, m + 5, (m,), generator=g, device="cuda").to(torch.int32)
    valid, keys, again = rows - 100, *(torch.zeros(m, dtype=torch.int64, device="cuda") for _ in "ab")
    y = ctx.marlin_gemm(x, w.words, w.scales, epi="argmax", xrows=order, keys=keys, n_valid=valid)
    assert torch.equal(y, ctx.marlin_gemm(x, w.words, w.scales, epi="argmax", xrows=order, keys=again, n_valid=valid))
    torch.cuda.synchronize()
    assert torch.equal(keys, again) and ctx.device_error() == 0
    a = y.cpu().numpy()
    assert (keys.cpu().numpy().view(np.uint64) == R.argmax_keys(a, valid)).all()
    x64, last = x[order.long()].double().cpu().numpy(), rows // 64 - 1
    groups = sorted({0, 1, last, *np.random.default_rng(m).integers(0, last, 5).tolist()})
    exact = {}
    for c in groups:
        q, s = R.unpack_marlin(w.words[:, 128 * c:128 * (c + 1)].cpu().numpy().view(np.uint32), w.scales[:, 64 * c:64 * (c + 1)].cpu().numpy())
        exact[c] = x64 @ ((q.astype(np.float64) - 8) * np.repeat(s.astype(np.float64), 128, 1)).T
    top = max(np.abs(e).max() for e in exact.values())
    for c, e in exact.items():
        assert np.abs(a[:, 64 * c:64 * (c + 1)] - e).max() < 1e-5 * top
    if m > 64:
        return
    rows3 = torch.arange(3, 3 + m, dtype=torch.int32, device="cuda")
    flat = ctx.marlin_gemm(x, w.words, w.scales, y=torch.zeros(m + 5, rows, device="cuda"), row0=3, m=m)
    assert torch.equal(flat[3:3 + m], ctx.marlin_gemm(x, w.words, w.scales, xrows=rows3)) and not flat[:3].any() and not flat[3 + m:].any()
    gl = ctx.marlin_gemm(x, w.words, w.scales, epi="silu", y=torch.zeros(m + 5, rows // 2, dtype=torch.float16, device="cuda"), row0=3, m=m)
    assert torch.equal(gl[3:3 + m], ctx.marlin_gemm(x, w.words, w.scales, epi="silu", xrows=rows3))
    gate, up = (t.double().reshape(m, -1) for t in flat[3:3 + m].view(m, rows // 16, 2, 8).unbind(2))
    want = gate / (1 + torch.exp(-gate)) * up   # (of the f32 sums: the f16 result falls on it or a neighbour)
    assert ((gl[3:3 + m].double() - want).abs() <= 2 ** -10 * want.abs() + 2 ** -23).all()
    assert ctx.device_error() == 0


@pytest.mark.parametrize("m,rows,cols", [(17, 256, 128), (40, 1024, 640), (64, 512, 1024)])
def test_few_rows_contiguous_from_row0(ctx, m, rows, cols):
    x, wdq, xd, wd, sd = make(rows, cols, True, 600 + m, m + 20)
    y = torch.zeros(m + 20, rows // 2, dtype=torch.float16, device="cuda")
    ctx.marlin_gemm(xd, wd, sd, epi="silu", y=y, row0=7, m=m)
    p = torch.zeros(m + 20, rows, device="cuda")
    keys = torch.zeros(m + 20, dtype=torch.int64, device="cuda")
    ctx.marlin_gemm(xd, wd, sd, epi="argmax", y=p, row0=7, m=m, keys=keys)
    torch.cuda.synchronize()
    assert ctx.device_error() == 0
    want = R.marlin_gemm(x[7:7 + m], wdq, "silu").astype(np.float32)
    a, b = y.float().cpu().numpy(), p.cpu().numpy()
    # (the f32 sums agree to 1e-5; the f16 result may fall on the neighbouring value)
    assert np.abs(a[7:7 + m] - want).max() <= 2 ** -10 * np.abs(want).max()
    assert np.all(a[:7] == 0) and np.all(a[7 + m:] == 0) and np.all(b[:7] == 0) and np.all(b[7 + m:] == 0)
    got = keys.cpu().numpy().view(np.uint64)
    assert (got[7:7 + m] == R.argmax_keys(b[7:7 + m], rows)).all() and np.all(got[:7] == 0) and np.all(got[7 + m:] == 0)


@pytest.mark.parametrize("m", [17, 32, 33, 64, 65, 97, 256, 257, 333])
def test_token_tile_widths_and_zero_points(ctx, m):
    """The tile's width follows the row count (32, 64, 96, 128, 256, 2 x 160, 2 x 192 tokens) of zero-point matrices, which take
    the prompt-sized product from 17 rows on."""
    g = synth.gen(700 + m)
    x = synth.activations(m, 384, g)
    codes, sc = synth.int4_matrix(512, 384, g)
    zeros = np.random.default_rng(m).integers(4, 13, (512, 3)).astype(np.uint8)
    words, s16 = host.pack_marlin(codes, sc, zeros=zeros)
    q, s = R.unpack_marlin(words, s16[:3])
    off = R.unpack_marlin(words, s16[3:])[1]
    dev = lambda a: torch.from_numpy(a).cuda()
    sd = dev(s16.view(np.int16)).view(torch.float16)
    y = ctx.marlin_gemm(dev(x), dev(words.view(np.int32)), sd, zp=True)
    torch.cuda.synchronize()
    assert ctx.device_error() == 0
    want = R.marlin_gemm(x, R.dequant_z(q, s, off))
    assert np.abs(y.cpu().numpy() - want).max() < 1e-5 * np.abs(want).max()
