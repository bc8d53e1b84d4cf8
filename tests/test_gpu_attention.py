"""Paged multi-query attention against the CPU oracle, plus the bit-equality grid of the reference's
kernel-vs-gather probe (crates/kiln-engine/tests/paged_attn.rs:40-52, 175-182) re-aimed at this
backend's invariant: verify row j (query length k+1) carries the bits of the one-row decode at the
same position, for permuted block tables, ragged tails and contexts that straddle chunk boundaries.
"""
import numpy as np
import pytest
import torch

from kiln_b200 import api
from oracle import oracle as O
from tests.conftest import cosine, parity

pytestmark = pytest.mark.gpu


def outlier_values(shape, seed):
    """xorshift-style outlier-heavy values: every 97th value x64 (paged_attn.rs:58-92 of the reference tests)."""
    g = torch.Generator().manual_seed(seed)
    v = torch.empty(shape).uniform_(-1, 1, generator=g)
    v.view(-1)[::97] *= 64.0
    return (v * 0.25).to(torch.bfloat16)


def fill_pools(ctx, spec, seed):
    """Identical random K/V content in a device pool set and an oracle pool set."""
    kv = api.PagedKv(ctx, spec)
    okv = O.OracleKv(spec.layers, spec.kv_heads, spec.head_dim, spec.num_blocks, spec.block_size)
    arr = okv.array()
    data = outlier_values(arr.shape, seed)
    arr[...] = data.view(torch.int16).numpy().view(np.uint16)
    per_block = spec.layers * 2 * spec.kv_heads * spec.block_size * spec.head_dim * 2
    for b in range(spec.num_blocks):
        # kc_kv_write_block payload: per layer the K rows then the V rows (paged.rs:280-304)
        payload = arr[:, :, b].tobytes()
        assert len(payload) == per_block
        kv.write_block_bytes(b, payload)
    return kv, okv


GRID = [
    # (head_dim, heads, kv_heads, block_size, [(len, offset), ...], softcap, window)
    (128, 8, 2, 16, [(6, 40)], 0.0, 0),                       # one verify segment, gqa 4
    (128, 8, 2, 16, [(1, 0), (1, 15), (1, 16), (1, 511), (1, 512), (1, 1300)], 0.0, 0),   # decode rows around tile/chunk edges
    (128, 8, 2, 16, [(6, 506), (6, 510), (5, 1020), (6, 1023)], 0.0, 0),     # verify segments straddling chunk boundaries
    (64, 8, 2, 32, [(5, 100), (5, 33), (1, 64)], 0.0, 0),     # head_dim 64, 32-token blocks
    (128, 7, 1, 16, [(5, 200), (5, 7)], 0.0, 0),              # gqa 7 (3 row tiles)
    (128, 8, 1, 16, [(5, 90)], 0.0, 0),                       # gqa 8
    (256, 4, 2, 16, [(4, 70), (4, 600)], 50.0, 0),            # gemma-2 geometry with softcap
    (256, 4, 2, 16, [(4, 70), (4, 600)], 50.0, 48),           # + sliding window
    (128, 8, 2, 16, [(40, 0), (23, 100)], 0.0, 0),            # prefill-shaped segments (several work items each)
    (128, 8, 2, 64, [(6, 700), (1, 130)], 0.0, 0),            # 64-token blocks (four tiles per block)
    (128, 8, 2, 128, [(6, 1100)], 0.0, 0),                    # 128-token blocks, three chunks
    (128, 8, 2, 16, [(6, 1500), (6, 300)], 0.0, 600),         # a window that ends inside an earlier chunk, head_dim 128
]


def build_seqs(segs, block_size, num_blocks, seed):
    rng = np.random.default_rng(seed)
    perm = rng.permutation(num_blocks)      # permuted block tables
    at = 0
    out = []
    for (ln, off) in segs:
        nb = (off + ln + block_size - 1) // block_size
        out.append(api.SeqStep(ln, off, ln, [int(x) for x in perm[at:at + nb]]))
        at += nb
    return out


@pytest.mark.parametrize("hd,heads,kvh,bs,segs,softcap,window", GRID)
def test_matches_oracle(ctx, hd, heads, kvh, bs, segs, softcap, window):
    nb = sum((off + ln + bs - 1) // bs for ln, off in segs) + 3
    spec = api.KvSpec(2, kvh, hd, nb, bs)
    kv, okv = fill_pools(ctx, spec, 11)
    seqs = build_seqs(segs, bs, nb, 5)
    n = sum(s.len for s in seqs)
    q = outlier_values((n, heads, hd), 7)
    scale = hd ** -0.5
    want = O.paged_attention(okv, 1, q, seqs, scale, softcap, window)
    got = api.paged_attention(ctx, kv, 1, q.cuda(), seqs, scale, softcap, window).cpu()
    label = f"attention D{hd} Hq{heads} Hkv{kvh} bs{bs} cap{softcap} win{window} {len(segs)} segs"
    if softcap > 0:
        # The reference's softcap attention rounds to bf16 after every op (nn.rs:497-580) and the oracle follows it; on
        # these outlier-heavy inputs its scores reach the cap (50), where one bf16 spacing is 0.25 and moves a
        # probability by e^0.25. The kernel keeps the scores in fp32, so the distance to the oracle here is the
        # oracle's own rounding noise; the bar for this op is 2e-2 of the output magnitude. (On model activations the
        # Gemma-2 forward is held to the flat logits bar in test_gpu_forward.py.)
        assert parity(label, got, want, bar=2e-2 * max(1.0, float(want.float().abs().max())))
    else:
        assert parity(label, got, want)
    assert ctx.device_status() == 0


@pytest.mark.parametrize("hd,heads,kvh,bs", [(128, 8, 2, 16), (64, 8, 2, 32), (128, 7, 1, 16), (256, 4, 2, 16)])
def test_verify_rows_carry_decode_bits(ctx, hd, heads, kvh, bs):
    """Row j of a (k+1)-row segment == the one-row launch at the same position, bit for bit, also when
    other sequences share the launch."""
    offsets = [3, 250, 509, 1019, 1500]
    k1 = 6
    nb = sum((o + k1 + bs - 1) // bs for o in offsets) + 2
    spec = api.KvSpec(1, kvh, hd, nb, bs)
    kv, _ = fill_pools(ctx, spec, 21)
    seqs = build_seqs([(k1, o) for o in offsets], bs, nb, 9)
    n = k1 * len(offsets)
    q = outlier_values((n, heads, hd), 8).cuda()
    scale = hd ** -0.5
    batched = api.paged_attention(ctx, kv, 0, q, seqs, scale).cpu()
    row = 0
    for s in seqs:
        for j in range(s.len):
            one = api.paged_attention(ctx, kv, 0, q[row:row + 1], [api.SeqStep(1, s.offset + j, 1, s.blocks)], scale).cpu()
            assert torch.equal(one.view(torch.int16), batched[row:row + 1].view(torch.int16)), \
                f"offset {s.offset} row {j}: verify row differs from decode row"
            row += 1


@pytest.mark.parametrize("hd,heads,kvh,softcap,window", [
    (64, 8, 2, 0.0, 0), (128, 8, 2, 0.0, 0), (128, 8, 2, 20.0, 300), (256, 4, 2, 50.0, 0), (256, 4, 2, 0.0, 90),
    (128, 7, 1, 0.0, 0), (64, 33, 1, 0.0, 0), (128, 64, 1, 0.0, 0), (256, 40, 1, 30.0, 700), (64, 1, 1, 0.0, 0), (128, 64, 1, 7.0, 513)])
@pytest.mark.parametrize("scale", [1.0, -0.5])
def test_prompt_rows_carry_decode_bits(ctx, hd, heads, kvh, softcap, window, scale):
    """The rows of a prompt's piece (more than 64 rows a unit: a thread holds a row) against the same rows a few at a time (a
    thread holds a key): the same bits, on both sides of tile and chunk edges, with 1 to 64 rows a unit."""
    gqa, bs = heads // kvh, 16
    start, length = 480, 80
    nb = (start + length + bs - 1) // bs
    kv, _ = fill_pools(ctx, api.KvSpec(1, kvh, hd, nb, bs), 41)
    blocks = build_seqs([(length, start)], bs, nb, 42)[0].blocks
    q = outlier_values((length, heads, hd), 43).cuda()
    scale *= hd ** -0.5
    whole = api.paged_attention(ctx, kv, 0, q, [api.SeqStep(length, start, length, blocks)], scale, softcap, window).cpu()
    for at, rows in [(0, 1), (27, min(53, 64 // gqa)), (31, 1), (32, 1), (length - 64 // gqa, 64 // gqa), (30, max(1, 32 // gqa)), (29, max(1, 17 // gqa))]:
        few = api.paged_attention(ctx, kv, 0, q[at: at + rows].contiguous(), [api.SeqStep(rows, start + at, rows, blocks)], scale, softcap, window).cpu()
        assert torch.equal(few.view(torch.int16), whole[at: at + rows].view(torch.int16)), f"rows {at} .. {at + rows}"
    assert ctx.device_status() == 0


@pytest.mark.parametrize("hd,heads,kvh,bs,layers", [(128, 8, 2, 16, 3), (64, 8, 2, 32, 2), (256, 4, 2, 16, 2)])
def test_one_operation_per_tile_pair_matches_the_slab_loads(ctx, monkeypatch, hd, heads, kvh, bs, layers):
    """A pool created with KILN_KV_MAP_2D=1 is read with one TMA operation per 64-feature slab of 8 keys, the default with one
    5-D operation per 16 keys of K or of V: the same shared-memory image, so the same bits, in every layer."""
    segs = [(6, 40), (1, 511), (6, 1020), (5, 7)]
    nb = sum((off + ln + bs - 1) // bs for ln, off in segs) + 2
    spec = api.KvSpec(layers, kvh, hd, nb, bs)
    kv4, _ = fill_pools(ctx, spec, 31)
    monkeypatch.setenv("KILN_KV_MAP_2D", "1")
    kv2, _ = fill_pools(ctx, spec, 31)
    monkeypatch.delenv("KILN_KV_MAP_2D")
    seqs = build_seqs(segs, bs, nb, 6)
    n = sum(s.len for s in seqs)
    q = outlier_values((n, heads, hd), 12).cuda()
    for layer in range(layers):
        a = api.paged_attention(ctx, kv4, layer, q, seqs, hd ** -0.5).cpu()
        b = api.paged_attention(ctx, kv2, layer, q, seqs, hd ** -0.5).cpu()
        assert torch.equal(a.view(torch.int16), b.view(torch.int16)), f"layer {layer}"
    assert ctx.device_status() == 0


@pytest.mark.parametrize("hd,heads,kvh,softcap,window", [(128, 8, 4, 0.0, 0), (64, 16, 4, 0.0, 700), (128, 8, 8, 30.0, 0)])
def test_units_of_whole_rows_carry_the_bits_of_single_chunks(ctx, hd, heads, kvh, softcap, window):
    """Many long sequences in one step: a unit holds all chunks of its rows and merges them itself. One sequence alone: a
    unit per chunk, merged by the combine kernel. Same bits, with lengths on both sides of tile and chunk edges."""
    check_whole_rows(ctx, hd, heads, kvh, 3, softcap, window)


@pytest.mark.parametrize("hd,heads,kvh,rows,softcap,window", [
    # a key per thread: two halves of the features, 32 rows and less, then 33 to 64
    (256, 8, 4, 3, 0.0, 0), (256, 8, 4, 3, 50.0, 700), (256, 8, 4, 16, 0.0, 0), (256, 8, 4, 17, 0.0, 700), (256, 16, 4, 16, 30.0, 0),
    (128, 16, 4, 9, 30.0, 0), (128, 16, 4, 16, 30.0, 600), (64, 16, 4, 11, 20.0, 0), (64, 16, 4, 16, 20.0, 0),
    # a row per thread
    (128, 8, 4, 40, 0.0, 0), (128, 8, 4, 40, 30.0, 700), (64, 8, 4, 40, 0.0, 700), (64, 16, 4, 11, 0.0, 0)])
def test_units_of_whole_rows_of_many_rows(ctx, hd, heads, kvh, rows, softcap, window):
    """The same with up to 64 rows a unit and more, and at head size 256, which the kernel with a key per thread alone has
    units of whole rows of."""
    check_whole_rows(ctx, hd, heads, kvh, rows, softcap, window)


def check_whole_rows(ctx, hd, heads, kvh, rows, softcap, window):
    rng = np.random.default_rng(3)
    # 74 sequences fill whole rounds of 148 CTAs: the most loaded one has 0.82 of what whole rows are allowed. With the
    # window, key 511 is seen by the first row of 1210 and not by its second: a chunk that is masked for some rows.
    lens = [511, 512, 513, 1023, 1024, 1151, 1210, 1537] + [int(v) for v in rng.integers(600, 1600, 66)]
    bs = 16
    nb = sum((n + rows + bs - 1) // bs for n in lens)
    kv = api.PagedKv(ctx, api.KvSpec(1, kvh, hd, nb, bs))
    data = outlier_values((64, kv.bytes_per_block() // 2), 51)
    for b in range(64):
        kv.write_block_bytes(b, data[b].view(torch.uint8).numpy().tobytes())
    for b in range(64, nb):
        kv.copy_block(b % 61, b)
    seqs = build_seqs([(rows, n) for n in lens], bs, nb, 52)
    q = outlier_values((rows * len(lens), heads, hd), 53).cuda()
    scale = hd ** -0.5
    before = ctx.launch_count()
    batched = api.paged_attention(ctx, kv, 0, q, seqs, scale, softcap, window).cpu()
    assert ctx.launch_count() == before + 1                                  # whole rows: nothing to merge afterwards
    for i, s in enumerate(seqs[:12]):
        before = ctx.launch_count()
        one = api.paged_attention(ctx, kv, 0, q[rows * i: rows * (i + 1)].contiguous(), [s], scale, softcap, window).cpu()
        assert ctx.launch_count() == before + 2                              # single chunks and the kernel that merges them
        assert torch.equal(one.view(torch.int16), batched[rows * i: rows * (i + 1)].view(torch.int16)), f"sequence {i}"
    assert ctx.device_status() == 0


@pytest.mark.parametrize("gain", [0.05, 1.0, 8.0, 60.0])
def test_softcap_over_its_range(ctx, gain):
    """Scores far below, around and beyond the cap against fp64. Bound: probabilities and output are rounded to bf16 (2^-9
    each, of outputs of order one); the cap itself adds under 1e-5."""
    hd, heads, kvh, bs, n = 128, 4, 1, 16, 300
    kv = api.PagedKv(ctx, api.KvSpec(1, kvh, hd, 20, bs))
    g = torch.Generator().manual_seed(61)
    k = torch.empty(19 * bs, hd).normal_(generator=g).to(torch.bfloat16)
    v = torch.empty(19 * bs, hd).normal_(generator=g).to(torch.bfloat16)
    for b in range(19):
        kv.write_block_bytes(b, torch.cat([k[b * bs: (b + 1) * bs].reshape(-1), v[b * bs: (b + 1) * bs].reshape(-1)]).view(torch.uint8).numpy().tobytes())
    q = (torch.empty(2, heads, hd).normal_(generator=g) * gain).to(torch.bfloat16)
    got = api.paged_attention(ctx, kv, 0, q.cuda(), [api.SeqStep(2, n, 2, list(range(19)))], hd ** -0.5, 5.0, 0).cpu().double()
    for t in range(2):
        x = q[t].double() @ k[: n + t + 1].double().T * hd ** -0.5
        want = torch.softmax(5.0 * torch.tanh(x / 5.0), -1) @ v[: n + t + 1].double()
        assert float((got.reshape(2, heads, hd)[t] - want).abs().max()) < 2 ** -8 * max(1.0, float(want.abs().max()))
    assert ctx.device_status() == 0


@pytest.mark.parametrize("scale", [0.0, -0.125, -4.0, 1e-3])
@pytest.mark.parametrize("hd,softcap,window", [(64, 0.0, 0), (128, 5.0, 0), (256, 3.0, 40)])
def test_any_scale(ctx, scale, hd, softcap, window):
    """Scales that turn the order of the scores round or make them all equal, against fp64, with keys on both sides of the
    mask in the last tile. Bound: the test above's."""
    heads, kvh, bs, n, rows = 4, 1, 16, 300, 3
    kv = api.PagedKv(ctx, api.KvSpec(1, kvh, hd, 20, bs))
    g = torch.Generator().manual_seed(71)
    k = torch.empty(19 * bs, hd).normal_(generator=g).to(torch.bfloat16)
    v = torch.empty(19 * bs, hd).normal_(generator=g).to(torch.bfloat16)
    for b in range(19):
        kv.write_block_bytes(b, torch.cat([k[b * bs: (b + 1) * bs].reshape(-1), v[b * bs: (b + 1) * bs].reshape(-1)]).view(torch.uint8).numpy().tobytes())
    q = torch.empty(rows, heads, hd).normal_(generator=g).to(torch.bfloat16)
    got = api.paged_attention(ctx, kv, 0, q.cuda(), [api.SeqStep(rows, n, rows, list(range(19)))], scale, softcap, window).cpu().double()
    for t in range(rows):
        first = max(0, n + t - window + 1) if window else 0
        x = q[t].double() @ k[first: n + t + 1].double().T * scale
        if softcap:
            x = softcap * torch.tanh(x / softcap)
        want = torch.softmax(x, -1) @ v[first: n + t + 1].double()
        assert float((got.reshape(rows, heads, hd)[t] - want).abs().max()) < 2 ** -8 * max(1.0, float(want.abs().max()))
    assert ctx.device_status() == 0


def test_softcap_of_scores_that_are_not_finite(ctx):
    """Under the cap an infinite score is plus or minus the cap, also where every key that a row sees has one; a NaN score
    makes the rows NaN that see it, and no other."""
    hd, heads, kvh, bs, n, cap = 64, 2, 1, 16, 180, 4.0
    g = torch.Generator().manual_seed(81)
    k = torch.empty(12 * bs, hd).normal_(generator=g) * 6
    v = torch.empty(12 * bs, hd).normal_(generator=g).to(torch.bfloat16)
    k[40], k[50] = 3e38, -3e38
    k[140:144] = -3e38
    k[182] = float("nan")
    k = k.to(torch.bfloat16)
    kv = api.PagedKv(ctx, api.KvSpec(1, kvh, hd, 12, bs))
    for b in range(12):
        kv.write_block_bytes(b, torch.cat([k[b * bs: (b + 1) * bs].reshape(-1), v[b * bs: (b + 1) * bs].reshape(-1)]).view(torch.uint8).numpy().tobytes())
    q = (torch.empty(5, heads, hd).uniform_(0.5, 1.5, generator=g)).to(torch.bfloat16)

    def check(offset, rows, window):
        got = api.paged_attention(ctx, kv, 0, q[:rows].cuda(), [api.SeqStep(rows, offset, rows, list(range(12)))], hd ** -0.5, cap, window)
        got = got.cpu().double().reshape(rows, heads, hd)
        for t in range(rows):
            first = max(0, offset + t - window + 1) if window else 0
            x = torch.nan_to_num(q[t].double() @ k[first: offset + t + 1].double().T, nan=float("nan")) * hd ** -0.5
            x = torch.where(x.abs() > 1e38, x.sign() * float("inf"), x)          # sums of fp32 products beyond its range
            want = torch.softmax(cap * torch.tanh(x / cap), -1) @ v[first: offset + t + 1].double()
            if offset + t >= 182:
                assert bool(torch.isnan(got[t]).all())
            else:
                assert float((got[t] - want).abs().max()) < 2 ** -8 * max(1.0, float(want.abs().max()))

    check(n, 5, 0)      # rows 0 and 1 before the NaN, 2 .. 4 from it on
    check(143, 3, 4)    # row 0 sees four keys of score -inf and no other
    assert ctx.device_status() == 0


@pytest.mark.parametrize("hd,batch,offset", [(64, 2, 40), (128, 2, 40), (256, 2, 40), (64, 1, 1300), (128, 1, 1300), (256, 1, 1300), (64, 148, 700), (128, 148, 700)])
def test_output_off_a_vector_boundary(ctx, hd, batch, offset):
    """The C entry point writes to any bf16 address: rows of one chunk, chunks merged by the second kernel, whole rows."""
    import ctypes as C
    from kiln_b200 import _lib as L
    heads, kvh, bs, rows = 4, 1, 16, 2
    need = (offset + rows + bs - 1) // bs
    kv = api.PagedKv(ctx, api.KvSpec(1, kvh, hd, need, bs))
    data = outlier_values((need, kv.bytes_per_block() // 2), 95)
    for b in range(need):
        kv.write_block_bytes(b, data[b].view(torch.uint8).numpy().tobytes())
    seqs = [api.SeqStep(rows, offset, rows, list(range(need)))] * batch
    q = outlier_values((rows * batch, heads, hd), 96).cuda()
    want = api.paged_attention(ctx, kv, 0, q, seqs, hd ** -0.5)
    p = api._PackedStep(api.StepBatch([0] * (rows * batch), seqs))
    for shift in (1, 2, 4):
        room = torch.full((want.numel() + 16,), 7.0, dtype=torch.bfloat16, device="cuda")
        torch.cuda.synchronize()
        api.check(L.lib().kc_paged_attention(ctx._h, kv._h, 0, q.data_ptr(), rows * batch, heads, p.seq_arr, p.n_seqs, hd ** -0.5, 0.0, 0,
                                             C.c_void_p(room.data_ptr() + 2 * shift)))
        assert torch.equal(room[shift: shift + want.numel()].view(torch.int16), want.view(-1).view(torch.int16))
        assert bool((room[:shift] == 7).all()) and bool((room[shift + want.numel():] == 7).all())
    assert ctx.device_status() == 0


@pytest.mark.parametrize("hd,batch,offset", [(64, 1, 40), (128, 1, 40), (256, 1, 40), (64, 1, 1300), (128, 1, 1300), (256, 1, 1300), (64, 148, 700), (128, 148, 700)])
def test_rows_are_divided_by_their_sums(ctx, hd, batch, offset):
    """Seven keys of equal weight and whole numbers: sums and weights are exact, and the quotients lie half way between two
    bf16 numbers, where a reciprocal that is rounded before the product shows. In every form a row is finished in: one
    chunk, chunks merged by the second kernel, whole rows. Values of -0 come out as +0 in each of them."""
    bs, window = 16, 7
    need = (offset + 1 + bs - 1) // bs
    kv = api.PagedKv(ctx, api.KvSpec(1, 1, hd, need, bs))
    t = torch.arange(hd) % 40 * 2 + 343                          # odd, of 9 bits: the means of seven bf16 numbers
    v = torch.zeros(need * bs, hd)
    first = offset - window + 1
    base = (t - 255) // 6 - ((t - 255) // 6 + 1) % 2             # 255 and six even numbers a little above the mean
    for j in range(6):
        v[first + j] = (t + base + 2 * (t - 255 - 6 * base > 2 * j)).float()
    v[first + 6] = 255
    assert torch.equal(v[first: first + 7].sum(0), 7.0 * t) and torch.equal(v, v.to(torch.bfloat16).float())
    want = t.to(torch.bfloat16)
    v[:, hd - 1] = -0.0
    want[hd - 1] = 0.0
    k = torch.zeros(need * bs, hd)
    for b in range(need):
        kv.write_block_bytes(b, torch.cat([k[b * bs: (b + 1) * bs].reshape(-1), v[b * bs: (b + 1) * bs].reshape(-1)]).to(torch.bfloat16).view(torch.uint8).numpy().tobytes())
    seqs = [api.SeqStep(1, offset, 1, list(range(need)))] * batch
    got = api.paged_attention(ctx, kv, 0, torch.ones(batch, 2, hd, dtype=torch.bfloat16, device="cuda"), seqs, hd ** -0.5, 0.0, window).cpu()
    assert torch.equal(got.view(batch * 2, hd).view(torch.int16), want.expand(batch * 2, hd).contiguous().view(torch.int16))
    assert ctx.device_status() == 0


@pytest.mark.parametrize("hd,keys", [(64, 50), (64, 700), (128, 200), (128, 1100), (256, 90), (256, 600)])
@pytest.mark.parametrize("gain", [0.3, 1.0, 3.0])
def test_error_is_that_of_the_output(ctx, hd, keys, gain):
    """Against fp64 the error is what rounding the rows to bf16 makes: 2^-7 / sqrt(12) of a value's power of two, 1.64e-3 of
    the norm of normally distributed values (the mean of their squares is 1.9 of that of their powers of two), with 2^-16
    for the probabilities. With those rounded to bf16 it was 1.7 to 2.3e-3. Bound: 4 % above the first for what 16000
    values scatter."""
    heads, kvh, bs, rows = 16, 4, 16, 8
    need = (keys + rows + bs - 1) // bs
    g = torch.Generator().manual_seed(97)
    k = torch.empty(need, kvh, bs, hd).normal_(generator=g).to(torch.bfloat16)
    v = torch.empty(need, kvh, bs, hd).normal_(generator=g).to(torch.bfloat16)
    kv = api.PagedKv(ctx, api.KvSpec(1, kvh, hd, need, bs))
    for b in range(need):
        kv.write_block_bytes(b, torch.cat([k[b].reshape(-1), v[b].reshape(-1)]).view(torch.uint8).numpy().tobytes())
    q = (torch.empty(rows, heads, hd).normal_(generator=g) * gain).to(torch.bfloat16)
    got = api.paged_attention(ctx, kv, 0, q.cuda(), [api.SeqStep(rows, keys, rows, list(range(need)))], hd ** -0.5).cpu().double().view(rows, heads, hd)
    kf, vf = (t.permute(1, 0, 2, 3).reshape(kvh, -1, hd).double() for t in (k, v))
    err = norm = 0.0
    for t in range(rows):
        x = torch.einsum("hgd,hkd->hgk", q[t].double().view(kvh, -1, hd), kf[:, : keys + t + 1]) * hd ** -0.5
        want = torch.einsum("hgk,hkd->hgd", torch.softmax(x, -1), vf[:, : keys + t + 1]).reshape(heads, hd)
        err += float((got[t] - want).square().sum())
        norm += float(want.square().sum())
    assert (err / norm) ** 0.5 < 1.71e-3
    assert ctx.device_status() == 0


def test_softcap_is_exact_to_a_rounding(ctx):
    """The cap's relative error, brought out by a cap of 2^20: two keys whose scores differ by a few units before the cap,
    weights read off one-hot values. Bound of a pair's log ratio: 1.1e-7 of either capped score below 0.75 caps, 1.7e-7
    above, and the two outputs' rounding to bf16 (2^-8 together)."""
    hd, kvh, bs, n, cap = 64, 8, 16, 400, 2.0 ** 20
    g = torch.Generator().manual_seed(99)
    y = torch.empty(n, kvh).uniform_(0.05, 2.5, generator=g)
    s = (y * cap).to(torch.bfloat16).double()
    y = s / cap
    d = torch.ceil(torch.empty(n, kvh).uniform_(0.2, 1.5, generator=g).double() / (1 - torch.tanh(y) ** 2)).to(torch.bfloat16).double()
    k = torch.zeros(n, kvh, bs, hd)
    k[:, :, 0, 0], k[:, :, 1, 0], k[:, :, 1, 1] = s.float(), s.float(), d.float()
    v = torch.zeros(n, kvh, bs, hd)
    v[:, :, 0, 0] = v[:, :, 1, 1] = 1
    kv = api.PagedKv(ctx, api.KvSpec(1, kvh, hd, n, bs))
    for b in range(n):
        kv.write_block_bytes(b, torch.cat([k[b].reshape(-1), v[b].reshape(-1)]).to(torch.bfloat16).view(torch.uint8).numpy().tobytes())
    q = torch.zeros(n, kvh, hd, dtype=torch.bfloat16)
    q[:, :, :2] = 1
    got = api.paged_attention(ctx, kv, 0, q.cuda(), [api.SeqStep(1, 1, 1, [b]) for b in range(n)], 1.0, cap).cpu().double().view(n, kvh, hd)
    ratio = torch.log(got[:, :, 1] / got[:, :, 0])
    want = cap * (torch.tanh((s + d) / cap) - torch.tanh(y))
    bound = torch.where(y < 0.75, 1.1e-7, 1.7e-7) * 2 * cap * torch.tanh(y) + 2 ** -8
    over = (ratio - want).abs() / bound
    assert float(over.max()) < 1, f"{float(over.max()):.2f} of the bound at {float(y.view(-1)[int(over.argmax())]):.3f} caps"
    assert ctx.device_status() == 0


@pytest.mark.parametrize("hd,heads,kvh,bs", [(128, 8, 2, 16), (64, 8, 2, 32), (256, 4, 2, 16)])
def test_slab_loads_of_prompt_rows(ctx, monkeypatch, hd, heads, kvh, bs):
    """The kernel with a row per thread over a pool of KILN_KV_MAP_2D=1: a slab of 8 keys an operation against 16 keys of K
    and V, the same bits."""
    segs = [(70, 500), (40, 0), (6, 1020)]
    nb = sum((off + ln + bs - 1) // bs for ln, off in segs) + 2
    spec = api.KvSpec(2, kvh, hd, nb, bs)
    kv5, _ = fill_pools(ctx, spec, 33)
    monkeypatch.setenv("KILN_KV_MAP_2D", "1")
    kv2, _ = fill_pools(ctx, spec, 33)
    monkeypatch.delenv("KILN_KV_MAP_2D")
    seqs = build_seqs(segs, bs, nb, 6)
    q = outlier_values((sum(s.len for s in seqs), heads, hd), 13).cuda()
    for layer in range(2):
        a, b = (api.paged_attention(ctx, kv, layer, q, seqs, hd ** -0.5).cpu() for kv in (kv5, kv2))
        assert torch.equal(a.view(torch.int16), b.view(torch.int16)), f"layer {layer}"
    assert ctx.device_status() == 0


@pytest.mark.parametrize("hd", [64, 128, 256])
@pytest.mark.parametrize("cap", [0.0, 4.0])
def test_prompt_rows_with_scores_that_are_not_finite(ctx, hd, cap):
    """Infinite and NaN scores in the kernel with a row per thread (80 rows a unit) against the rows one at a time (a key per
    thread): the same rows are NaN, the others have the same bits."""
    heads, kvh, bs, n, rows = 2, 1, 16, 140, 40
    g = torch.Generator().manual_seed(83)
    k = torch.empty(12 * bs, hd).normal_(generator=g) * 6
    v = torch.empty(12 * bs, hd).normal_(generator=g).to(torch.bfloat16)
    k[40], k[140:144] = -3e38, -3e38
    k[160] = 3e38
    k[172] = float("nan")
    k = k.to(torch.bfloat16)
    kv = api.PagedKv(ctx, api.KvSpec(1, kvh, hd, 12, bs))
    for b in range(12):
        kv.write_block_bytes(b, torch.cat([k[b * bs: (b + 1) * bs].reshape(-1), v[b * bs: (b + 1) * bs].reshape(-1)]).view(torch.uint8).numpy().tobytes())
    q = (torch.empty(rows, heads, hd).uniform_(0.5, 1.5, generator=g)).to(torch.bfloat16).cuda()
    many = api.paged_attention(ctx, kv, 0, q, [api.SeqStep(rows, n, rows, list(range(12)))], hd ** -0.5, cap).cpu()
    one = torch.cat([api.paged_attention(ctx, kv, 0, q[t: t + 1].contiguous(), [api.SeqStep(1, n + t, 1, list(range(12)))], hd ** -0.5, cap).cpu() for t in range(rows)])
    assert torch.equal(torch.isnan(many), torch.isnan(one))
    assert not bool(torch.isnan(many[: 160 - n]).any()) and bool(torch.isnan(many[172 - n:]).all())
    assert torch.equal(torch.nan_to_num(many, nan=0.0).view(torch.int16), torch.nan_to_num(one, nan=0.0).view(torch.int16))
    assert ctx.device_status() == 0
