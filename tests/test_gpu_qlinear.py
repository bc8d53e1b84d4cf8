"""Affine-dequant GEMM (kc_quantized_matmul) against the CPU oracle.

Mirrors the reference's use of quantized_matmul (crates/kiln-models/src/nn.rs:79-102) and its
row-stability probe (nn.rs:301-327): row r of Y(M) must carry the bits of Y(1).
Tolerance is the north-star logits bar applied per layer: max-abs <= 2e-2, cosine >= 0.9999.
"""
import pytest
import torch

from kiln_b200 import api
from kiln_b200.synth import quantize_affine
from oracle import oracle as O
from tests.conftest import cosine, parity

pytestmark = pytest.mark.gpu

MAX_ABS, MIN_COS = 2e-2, 0.9999


def make(n, k, bits, group, seed):
    g = torch.Generator().manual_seed(seed)
    w = torch.empty(n, k).normal_(0, 0.02, generator=g)
    # outlier-heavy values like the reference's kernel probes (crates/kiln-engine/tests/paged_attn.rs:58-70)
    w.view(-1)[::97] *= 8.0
    return quantize_affine(w, bits, group)


def acts(m, k, seed):
    g = torch.Generator().manual_seed(seed)
    x = torch.empty(m, k).normal_(0, 1.0, generator=g)
    x.view(-1)[::97] *= 16.0
    return x.to(torch.bfloat16)


CASES = [
    # (N, K, bits, group, M)
    (256, 256, 4, 64, 5),          # tiny: one k-split
    (200, 512, 4, 64, 17),         # N not a multiple of the 128-row tile
    (384, 1024, 4, 32, 33),        # two groups per k-block
    (256, 1024, 4, 128, 6),        # a group spans two k-blocks
    (256, 512, 8, 32, 48),         # 8-bit
    (256, 448, 8, 64, 7),          # K = 7 k-blocks
    (1024, 4096, 4, 64, 192),      # the 8B attention-output shape at verify width: split-K engaged
    (2048, 2048, 4, 64, 320),      # two chunks of rows
    (512, 2048, 4, 64, 1),         # decode row
    (53248, 256, 8, 32, 100),      # 416 tiles of 8-bit records at 100 rows
]


@pytest.mark.parametrize("n,k,bits,group,m", CASES)
def test_matches_oracle(ctx, n, k, bits, group, m):
    p, s, b = make(n, k, bits, group, 1)
    x = acts(m, k, 2)
    O.set_weight_class(1)      # the tensor-core kernel's arithmetic class: w = bf16(q * scale + bias) first
    want = O.quantized_matmul(x, p, s, b, bits, group)
    O.set_weight_class(0)
    qw = api.QuantizedWeight(ctx, p.cuda(), s.cuda(), b.cuda(), bits, group)
    got = qw.matmul(x.cuda()).cpu()
    # 2e-2 flat below magnitude 4; above it one bf16 spacing of the value is added (outputs here reach 20+)
    assert parity(f"qlinear {n}x{k} w{bits}g{group} rows {m}", got, want, MAX_ABS, MIN_COS)
    assert ctx.device_status() == 0


@pytest.mark.parametrize("n,k,bits,group", [(1024, 4096, 4, 64), (256, 512, 8, 32), (4096, 1024, 4, 128)])
def test_rows_do_not_depend_on_batch_width(ctx, n, k, bits, group):
    """probe_row_stability (nn.rs:301-327) widened: every row of Y(M) is bit-identical to its M=1 result."""
    p, s, b = make(n, k, bits, group, 3)
    qw = api.QuantizedWeight(ctx, p.cuda(), s.cuda(), b.cuda(), bits, group)
    x = acts(320, k, 4).cuda()
    ref_rows = {r: qw.matmul(x[r:r + 1]).cpu() for r in (0, 1, 5, 31, 191, 319)}
    for m in (2, 5, 6, 32, 192, 320):
        y = qw.matmul(x[:m]).cpu()
        for r, want in ref_rows.items():
            if r < m:
                assert torch.equal(y[r:r + 1].view(torch.int16), want.view(torch.int16)), f"row {r} differs at M={m}"


STREAM_CASES = [
    # (N, K, bits, group, M): the weight-streaming lane, at most 8 rows
    (256, 256, 4, 64, 1),          # one k-split
    (200, 512, 4, 64, 5),          # N not a multiple of the 128-row tile
    (384, 1024, 4, 32, 8),         # two groups per k-block
    (256, 1024, 4, 128, 3),        # a group spans two k-blocks
    (256, 512, 8, 32, 8),          # 8-bit
    (256, 448, 8, 64, 7),          # K = 7 k-blocks: uneven k-splits
    (1024, 4096, 4, 64, 6),        # the 8B attention-output shape: several pieces per tile
    (28672, 4096, 4, 64, 8),       # the 8B gate_up shape
    (4099, 2048, 4, 64, 2),        # a ragged last tile
    (640, 14336, 4, 64, 4),        # the 8B down-projection depth: a tile's k-blocks spread over many CTAs
    (128256, 2048, 4, 64, 1),      # the 1B head: runs that cross two tile boundaries
]


@pytest.mark.parametrize("n,k,bits,group,m", STREAM_CASES)
def test_stream_lane_matches_oracle(ctx, n, k, bits, group, m):
    """kc_quantized_matmul_stream is of MLX's row-vector class (scale and bias applied per group to fp32 sums of
    x q and of x), the oracle's class 0; against the tensor-core lane (weights rounded to bf16 first) the distance is
    that of the two classes."""
    p, s, b = make(n, k, bits, group, 5)
    x = acts(m, k, 6)
    O.set_weight_class(0)
    want = O.quantized_matmul(x, p, s, b, bits, group)
    qw = api.QuantizedWeight(ctx, p.cuda(), s.cuda(), b.cuda(), bits, group)
    got = qw.matmul_stream(x.cuda()).cpu()
    assert parity(f"stream lane {n}x{k} w{bits}g{group} rows {m}", got, want, MAX_ABS, MIN_COS)
    tensor = qw.matmul(x.cuda()).cpu()
    # two arithmetic classes apart: the distance is printed, and held to what the oracle's own two classes differ by on
    # the same inputs (plus one bf16 spacing of the largest value for the kernels' accumulation orders)
    O.set_weight_class(1)
    want_tile = O.quantized_matmul(x, p, s, b, bits, group)
    O.set_weight_class(0)
    class_gap = float((want.float() - want_tile.float()).abs().max())
    spacing = 2.0 ** (torch.floor(torch.log2(want.float().abs().max())) - 7)
    parity(f"stream lane vs tensor lane {n}x{k} w{bits}g{group} rows {m}", got, tensor, 1e9, MIN_COS)
    gap = float((got.float() - tensor.float()).abs().max())
    print(f"oracle class 0 vs class 1: max-abs {class_gap:.4g}; lanes: {gap:.4g}")
    assert gap <= class_gap + 2 * float(spacing)
    assert cosine(got, tensor) >= MIN_COS
    assert ctx.device_status() == 0


GEMV_CASES = [
    # (N, K, bits, group, M): the small-weight lane of the same arithmetic
    (256, 256, 4, 64, 1),
    (200, 512, 4, 64, 5),          # N not a multiple of the 128-row tile
    (384, 1024, 4, 32, 8),         # two groups per k-block
    (256, 1024, 4, 128, 3),        # a group spans two k-blocks
    (256, 512, 8, 32, 8),          # 8-bit
    (256, 448, 8, 64, 7),          # K = 7 k-blocks: uneven runs
    (3072, 2048, 4, 64, 1),        # the 1B qkv shape
    (2048, 2048, 4, 64, 4),        # the 1B attention-output shape
    (16384, 2048, 4, 64, 1),       # the 1B gate_up shape: two runs per tile
    (2048, 8192, 4, 64, 8),        # the 1B down-projection depth: eight runs of 16 k-blocks
    (4099, 2048, 4, 64, 2),        # a ragged last tile
]


@pytest.mark.parametrize("n,k,bits,group,m", GEMV_CASES)
def test_small_weight_lane_matches_oracle_and_the_streaming_lane(ctx, n, k, bits, group, m):
    """kc_quantized_matmul_gemv against the oracle's row-vector class, and against the streaming kernel of the same
    class (they differ only in where a tile's k-blocks are cut, i.e. in fp32 summation order)."""
    p, s, b = make(n, k, bits, group, 15)
    x = acts(m, k, 16)
    O.set_weight_class(0)
    want = O.quantized_matmul(x, p, s, b, bits, group)
    qw = api.QuantizedWeight(ctx, p.cuda(), s.cuda(), b.cuda(), bits, group)
    got = qw.matmul_gemv(x.cuda()).cpu()
    assert parity(f"small-weight lane {n}x{k} w{bits}g{group} rows {m}", got, want, MAX_ABS, MIN_COS)
    stream = qw.matmul_stream(x.cuda()).cpu()
    spacing = 2.0 ** (torch.floor(torch.log2(want.float().abs().max())) - 7)
    assert float((got.float() - stream.float()).abs().max()) <= 2 * float(spacing)
    # a row's bits do not depend on how many rows ride the call
    if m > 1:
        one = qw.matmul_gemv(x[:1].cuda()).cpu()
        assert torch.equal(one.view(torch.int16), got[:1].view(torch.int16))
    assert ctx.device_status() == 0


def test_small_weight_lane_refuses_a_shape_it_cannot_hold(ctx):
    """224 k-blocks would need more than eight runs of what shared memory holds: the entry point says so."""
    p, s, b = make(640, 14336, 4, 64, 3)
    qw = api.QuantizedWeight(ctx, p.cuda(), s.cuda(), b.cuda(), 4, 64)
    message = None
    try:
        qw.matmul_gemv(acts(2, 14336, 4).cuda())
    except api.KcError as err:     # only the text is kept: a stored traceback would keep the weight alive past its context
        message = str(err)
    assert message and "does not fit" in message


def test_stream_lane_rows_do_not_depend_on_row_count(ctx):
    """Within the lane a row's bits do not depend on how many rows ride the call (1..8)."""
    p, s, b = make(1024, 4096, 4, 64, 7)
    qw = api.QuantizedWeight(ctx, p.cuda(), s.cuda(), b.cuda(), 4, 64)
    x = acts(8, 4096, 8).cuda()
    full = qw.matmul_stream(x).cpu()
    for m in (1, 2, 3, 5, 7):
        y = qw.matmul_stream(x[:m]).cpu()
        assert torch.equal(y.view(torch.int16), full[:m].view(torch.int16))
    one = qw.matmul_stream(x[5:6]).cpu()
    assert torch.equal(one.view(torch.int16), full[5:6].view(torch.int16))
    with pytest.raises(api.KcError, match="m = 9"):
        qw.matmul_stream(acts(9, 4096, 9).cuda())


@pytest.mark.parametrize("n,k,bits,group,m,gain", [
    (26700, 192, 4, 64, 33, 1.0),     # 209 tiles: the last team's second CTA has none; three k-blocks
    (26700, 64, 8, 64, 192, 1.0),     # one k-block
    (384, 1088, 4, 32, 192, 1.0),     # the most rows of one chunk, splits of 8 and 9 k-blocks: an odd number of them
    (384, 1088, 4, 32, 256, 1.0),     # the same in two chunks
    (384, 1088, 8, 32, 177, 1.0),     # 8-bit, rows past the activations' end inside the last group of 16
    (300, 512, 4, 64, 20, 200.0),     # scales of 0.5 and more: taken at 2^-shift of their size
    (300, 512, 8, 64, 20, 300.0),     # the same for 8 bits (scales of 1/32 and more)
    (300, 512, 4, 64, 20, 1e-30),     # scales near the smallest normal numbers
])
def test_stage_edges_and_scale_range(ctx, n, k, bits, group, m, gain):
    """The places where the pipeline's stages end unevenly, and the range of scales on both sides of the one from which on
    weights are taken at 2^-shift of their size. Bound: the GEMM's bar for outputs of order one; with another gain the outputs scale
    with it, so the inputs are scaled back by a power of two and the same bar holds."""
    g = torch.Generator().manual_seed(31)
    w = torch.empty(n, k).normal_(0, 0.02 * gain, generator=g)
    p, s, b = quantize_affine(w, bits, group)
    if gain > 1:
        assert float(s.float().max()) >= (0.5 if bits == 4 else 0.03125)
    if gain < 1e-20:
        s = (s.float() * 0 + 2.0 ** -110).to(torch.bfloat16)      # the quantiser's floor is far above such a gain
        b = (b.float().sign() * 2.0 ** -108).to(torch.bfloat16)
        shift = 2.0 ** 108
    else:
        shift = 2.0 ** -int(torch.log2(torch.tensor(gain)).round())
    x = (acts(m, k, 32).float() * shift).to(torch.bfloat16)
    O.set_weight_class(1)
    want = O.quantized_matmul(x, p, s, b, bits, group)
    O.set_weight_class(0)
    qw = api.QuantizedWeight(ctx, p.cuda(), s.cuda(), b.cuda(), bits, group)
    got = qw.matmul(x.cuda()).cpu()
    assert parity(f"qlinear {n}x{k} w{bits}g{group} rows {m} gain {gain:g}", got, want, MAX_ABS, MIN_COS)
    one = qw.matmul(x[m - 1:].cuda()).cpu()
    assert torch.equal(one.view(torch.int16), got[m - 1:].view(torch.int16))
    assert ctx.device_status() == 0


@pytest.mark.parametrize("n,k,bits,group,m", [
    (26700, 320, 4, 64, 193),     # two chunks, the last team's second tile missing
    (26700, 384, 4, 128, 1001),   # a last chunk of fewer rows than the others
    (384, 1088, 4, 32, 257),      # split along K
    (300, 512, 8, 64, 700),       # more rows than a slab of the split-K workspace
])
def test_row_chunks_carry_the_bits_of_few_rows(ctx, n, k, bits, group, m):
    """Rows are cut into chunks by a rule on the shape: a row's bits are those it has in a launch of its own."""
    p, s, b = make(n, k, bits, group, 41)
    qw = api.QuantizedWeight(ctx, p.cuda(), s.cuda(), b.cuda(), bits, group)
    x = acts(m, k, 42).cuda()
    full = qw.matmul(x).cpu()
    for r0, r1 in ((0, 1), (90, 131), (m - 70, m), (m - 1, m)):
        part = qw.matmul(x[r0:r1].contiguous()).cpu()
        assert torch.equal(part.view(torch.int16), full[r0:r1].view(torch.int16)), f"rows {r0}..{r1}"
    assert ctx.device_status() == 0


@pytest.mark.parametrize("n,k,bits,group,m,gain", [
    (384, 1088, 4, 32, 1201, 1.0),    # three tiles, splits of 8 and 9 k-blocks, a last chunk of few rows
    (4100, 2176, 4, 128, 1300, 1.0),  # several items a CTA, splits of 8 and 9 k-blocks, a ragged last tile
    (300, 1024, 4, 64, 1000, 200.0),  # scales of 0.5 and more: taken at 2^-shift of their size
    (4608, 3584, 8, 32, 1111, 1.0),
    (6144, 4096, 4, 64, 700, 1.0),    # three splits
    (1000, 1024, 8, 64, 5003, 1.0),
])
def test_many_rows_carry_the_bits_of_few(ctx, n, k, bits, group, m, gain):
    """Many rows: persistent CTAs, which take all splits of their tile and rows one after the other instead of leaving
    partials. A row's bits are those it has in a launch of few rows, where a split is a CTA of its own."""
    g = torch.Generator().manual_seed(43)
    p, s, b = quantize_affine(torch.empty(n, k).normal_(0, 0.02 * gain, generator=g), bits, group)
    qw = api.QuantizedWeight(ctx, p.cuda(), s.cuda(), b.cuda(), bits, group)
    x = acts(m, k, 44).cuda()
    full = qw.matmul(x).cpu()
    for r0, r1 in ((0, 1), (90, 131), (m // 2, m // 2 + 170), (m - 70, m), (m - 1, m)):
        part = qw.matmul(x[r0:r1].contiguous()).cpu()
        assert torch.equal(part.view(torch.int16), full[r0:r1].view(torch.int16)), f"rows {r0}..{r1}"
    assert ctx.device_status() == 0


@pytest.mark.parametrize("bits", [4, 8])
@pytest.mark.parametrize("scale", [129 / 2 ** 10, 129 / 2 ** 8])     # below and above the line from which on weights are taken at 2^-shift of their size
def test_weights_are_rounded_once(ctx, bits, scale):
    """A weight is q * scale + bias rounded to bf16 once: with a bias far below the last bit of a product that lies half way
    between two bf16 numbers, a rounding to fp32 in between loses it and the half way goes to the even one. Exact: one-hot
    rows bring the weights out as they are."""
    if bits == 8:
        scale /= 16
    n, k = 128, 64
    g = torch.Generator().manual_seed(91)
    q = torch.randint(0, 2 ** bits, (n, k), generator=g)
    q[:, 0], q[:, 1] = 3, 5                                            # 3 * 129 and 5 * 129 have 9 and 10 bits: half ways among them
    per = 32 // bits
    packed = (q.reshape(n, -1, per) << (torch.arange(per) * bits)).sum(-1)
    packed = torch.where(packed >= 2 ** 31, packed - 2 ** 32, packed).to(torch.int32)
    s = torch.full((n, 1), scale).to(torch.bfloat16)
    b = (torch.where(torch.arange(n) % 2 == 0, 1.0, -1.0) * 2.0 ** -34).reshape(n, 1).to(torch.bfloat16)
    exact = q.double() * s.double() + b.double()
    ulp = torch.exp2(torch.floor(torch.log2(exact.abs())) - 7)
    want = (torch.round(exact / ulp) * ulp).float()                    # half to even, of the exact value
    via_fp32 = exact.float().to(torch.bfloat16).float()
    assert not torch.equal(want, via_fp32)                             # the input tells the two apart
    qw = api.QuantizedWeight(ctx, packed.cuda(), s.cuda(), b.cuda(), bits, 64)
    got = qw.matmul(torch.eye(k).to(torch.bfloat16).cuda()).cpu().float().T
    assert torch.equal(got, want)
    assert ctx.device_status() == 0


def chunks_of_cut_pairs(n, k, m):
    """The library's rule for a weight of one chain of products, restated: the chunks of rows of a launch whose teams cut pairs of weight tiles
    between them, 0 where they have whole pairs."""
    teams, pairs, blocks = 74, (-(-n // 128) + 1) // 2, k // 64
    assert pairs * 10 >= 148 * 7
    best = None
    for per in (192, 160, 128, 96):
        if per - 32 >= m and per > 96:
            continue
        chunks = -(-m // per)
        whole, cut = -(-pairs * chunks // teams) * blocks, (pairs * blocks / teams + 20) * chunks
        cuts = chunks <= 3 and cut < whole
        cost = (cut if cuts else whole) * (max(300, 2 * per) + 20)
        if best is None or cost < best[0] * 0.995:
            best = cost, chunks if cuts else 0
    return best[1]


@pytest.mark.parametrize("n,k,bits,group,gain,cuts", [
    (28672, 4096, 4, 64, 1.0, {1: 1, 17: 1, 64: 1, 65: 1, 128: 1, 192: 1, 384: 2, 577: 0}),    # a pair and a half a team: two and three pairs of a run
    (28672, 4096, 8, 32, 300.0, {1: 1, 96: 1, 97: 1, 384: 2}),                                # .. at 2^-shift of its size
    (28665, 4160, 4, 32, 200.0, {5: 1, 80: 1, 150: 1, 383: 2}),                               # 65 k-blocks; rows that leave value by value
    (31744, 8192, 4, 64, 1.0, {33: 1, 576: 3}),                                               # all chunks that the workspace has room for
])
def test_teams_that_share_a_pair_carry_its_bits(ctx, n, k, bits, group, gain, cuts):
    """A team that has the end of a pair of weight tiles goes on from the sums of the one that has its start: one chain of products,
    whoever has it. The entry point without that workspace has whole pairs only; few rows, rows of a cluster, and two and three chunks."""
    g = torch.Generator(device="cuda").manual_seed(51)
    p, s, b = quantize_affine(torch.empty(n, k, device="cuda").normal_(0, 0.02 * gain, generator=g), bits, group)
    qw = api.QuantizedWeight(ctx, p, s, b, bits, group)
    x = acts(max(cuts), k, 52).cuda()
    want = torch.empty(max(cuts), n, dtype=torch.bfloat16, device="cuda")
    qw.matmul_static(torch.cat([x, x[:16]]), max(cuts), want)
    ctx.sync()
    for m, chunks in list(cuts.items()) + [(min(cuts), 1)]:
        assert chunks_of_cut_pairs(n, k, m) == chunks
        y = qw.matmul(x[:m])
        assert torch.equal(y.view(torch.int16), want[:m].view(torch.int16)), m
    assert ctx.device_status() == 0


@pytest.mark.parametrize("n,k,bits,group", [
    (384, 1088, 4, 32),           # splits of 8 and 9 k-blocks
    (4096, 2048, 8, 32),          # four splits, apart and in turn
    (11000, 256, 4, 64),          # not split
    (19000, 1088, 4, 64),         # not split, more pairs of tiles than teams
])
def test_even_and_odd_k_blocks_are_sums_of_their_own(ctx, n, k, bits, group):
    """Weights of fewer than 207 tiles: a split is two chains of products, its even and its odd k-blocks, half as long as one. Exact:
    a large value and its negative two k-blocks on cancel, and take what one sum would have had between them with it."""
    tiles, blocks = -(-n // 128), k // 64
    splits = 1 if 2 * tiles >= 148 else max(1, min(148 // tiles, 16, blocks // 8))
    packed = torch.full((n, k * bits // 32), 0x11111111 if bits == 4 else 0x01010101, dtype=torch.int32)
    one = torch.ones(n, k // group, dtype=torch.bfloat16)
    qw = api.QuantizedWeight(ctx, packed.cuda(), one.cuda(), (one * 0).cuda(), bits, group)
    rows = torch.arange(1100)
    x = torch.zeros(1100, k)
    for s in range(splits):
        at = blocks * s // splits * 64
        x[:, at], x[:, at + 64], x[:, at + 128] = 2.0 ** 30, (rows % 7 + 1).float(), -2.0 ** 30
    x = x.to(torch.bfloat16).cuda()
    want = ((rows % 7 + 1) * splits).float().reshape(-1, 1)
    for m in (1, 17, 64, 65, 130, 192, 320, 1100):
        assert torch.equal(qw.matmul(x[:m]).cpu().float(), want[:m].expand(m, n)), m
    assert ctx.device_status() == 0


@pytest.mark.parametrize("n,k", [(301, 512), (300, 1024), (4099, 4096), (9500, 256), (19501, 512)])
def test_rows_that_are_not_aligned_match_aligned_ones(ctx, n, k):
    """Widths that are no multiple of eight leave value by value, as y and as partials of splits: the same bits as the aligned weight that
    the rows are the first ones of, in lone CTAs and in pairs."""
    wide = (n + 127) // 128 * 128       # as many tiles, so the same splits and chains
    p, s, b = make(wide, k, 4, 64, 61)
    aligned = api.QuantizedWeight(ctx, p.cuda(), s.cuda(), b.cuda(), 4, 64)
    ragged = api.QuantizedWeight(ctx, p[:n].contiguous().cuda(), s[:n].contiguous().cuda(), b[:n].contiguous().cuda(), 4, 64)
    x = acts(321, k, 62).cuda()
    for m in (1, 9, 64, 121, 150, 250, 321):
        want, got = aligned.matmul(x[:m])[:, :n], ragged.matmul(x[:m])
        assert torch.equal(got.view(torch.int16), want.contiguous().view(torch.int16)), m
    assert ctx.device_status() == 0


@pytest.mark.parametrize("bits", [4, 8])
@pytest.mark.parametrize("large,small", [(100, -30), (20, -40), (30, -39), (127, -126), (-4, -120), (-4, -40)])
def test_scales_far_apart_are_exact(ctx, bits, large, small):
    """A weight with large scales is taken at a power of two less only where that is exact: rows of the largest and of far smaller scales
    and biases come out as q * scale + bias rounded once. Exact: one-hot rows bring the weights out as they are."""
    n, k = 256, 128
    g = torch.Generator().manual_seed(71)
    q = torch.randint(0, 2 ** bits, (n, k), generator=g)
    per = 32 // bits
    packed = (q.reshape(n, -1, per) << (torch.arange(per) * bits)).sum(-1)
    packed = torch.where(packed >= 2 ** 31, packed - 2 ** 32, packed).to(torch.int32)
    power = torch.full((n, 1), float(small), dtype=torch.float64)
    power[::7] = large - bits                                            # the largest product stays a bf16 number
    s = (torch.exp2(power) * (129 / 128)).expand(n, 2).to(torch.bfloat16).contiguous()
    b = (torch.exp2(power) * torch.where(torch.arange(n).reshape(n, 1) % 2 == 0, -5.0, 3.0)).expand(n, 2).to(torch.bfloat16).contiguous()
    exact = q.double() * s.double().repeat_interleave(64, 1) + b.double().repeat_interleave(64, 1)
    ulp = torch.exp2(torch.floor(torch.log2(exact.abs().clamp_min(2.0 ** -126))) - 7)
    want = (torch.round(exact / ulp) * ulp).float()                      # half to even, of the exact value
    qw = api.QuantizedWeight(ctx, packed.cuda(), s.cuda(), b.cuda(), bits, 64)
    got = qw.matmul(torch.eye(k).to(torch.bfloat16).cuda()).cpu().float().T
    assert torch.equal(got, want)
    assert ctx.device_status() == 0
