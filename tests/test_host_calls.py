"""What the library asks of the CUDA runtime, call by call, against a stand-in for it (fake_cudart.cpp): the order and kind
of launches, failures of allocations, limits of a launch. Needs no GPU; each test is a process of its own."""
import os
import subprocess
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent

PRELUDE = """
import ctypes as C
from kiln_b200 import _lib as L
fake = C.CDLL(None)
fake.fake_calls.restype = C.c_char_p
fake.fake_fail_above.argtypes = [C.c_size_t]
lib = C.CDLL(str(L.LIB_PATH))
for name, (res, args) in L._SIGNATURES.items():
    f = getattr(lib, name)
    f.restype, f.argtypes = res, args
def ok(rc):
    assert rc == 0, lib.kc_last_error()
def calls():
    out = fake.fake_calls().decode().splitlines()
    fake.fake_reset()
    return out
ctx = C.c_void_p()
ok(lib.kc_ctx_create(0, C.byref(ctx)))
kv = C.c_void_p()
ok(lib.kc_kv_create(ctx, 1, 2, 64, 80, 16, L.KC_BF16, C.byref(kv)))
room = C.create_string_buffer(1 << 20)
at = (C.addressof(room) + 255) // 256 * 256
table = (C.c_uint32 * 80)(*range(80))
def attention(lens, out=at, heads=4):
    seqs = (L.KcSeqStep * len(lens))(*[L.KcSeqStep(n, off, n, -(-(n + off) // 16), table) for n, off in lens])
    return lib.kc_paged_attention(ctx, kv, 0, at, sum(n for n, _ in lens), heads, seqs, len(lens), 0.125, 0.0, 0, out)
"""


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    so = tmp_path_factory.mktemp("fake") / "fake_cudart.so"
    subprocess.run(["g++", "-shared", "-fPIC", "-O1", "-I/usr/local/cuda/include", "-o", str(so), str(ROOT / "tests" / "fake_cudart.cpp")], check=True)
    return so


def run(fake, code, first=""):
    r = subprocess.run([sys.executable, "-c", first + PRELUDE + code], cwd=ROOT, env={**os.environ, "LD_PRELOAD": str(fake), "PYTHONPATH": str(ROOT)},
                       capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr


def test_attention_waits_for_its_metadata(fake):
    """The kernel behind the copy of a call's metadata reads it before it waits for the kernel ahead of it: it must be
    ordered behind the copy. The kernel that merges the chunks may start early."""
    run(fake, """
for lens in ([(3, 40)], [(1, 1000)]):       # one launch; chunks and the kernel that merges them
    fake.fake_reset()
    ok(attention(lens))
    seen = [c for c in calls() if c.startswith(("copy", "launch"))]
    assert seen[:2] == ["copy", "launch in order"], seen
    assert seen[2:] in ([], ["launch early"]), seen
assert seen[2:] == ["launch early"], seen
""")


def test_rope_waits_for_its_metadata(fake):
    """Positions, slots and a caller's frequencies are read before the wait for the kernel ahead: a single call's launch is
    ordered behind the copy that brings them, and behind the caller's own work."""
    run(fake, """
fake.fake_reset()
seqs = (L.KcSeqStep * 1)(L.KcSeqStep(3, 40, 3, 3, table))
ok(lib.kc_rope_kv_write(ctx, kv, 0, at, None, C.cast(at, C.POINTER(C.c_float)), 3, 4, 0, seqs, 1, at))
seen = [c for c in calls() if c.startswith(("copy", "launch"))]
assert seen == ["copy", "launch in order"], seen
""")


@pytest.mark.parametrize("dim", [1024, 2048, 4096, 8192])
def test_rms_norm_waits_for_its_weight(fake, dim):
    """The weight is read before the kernel ahead has finished, and a caller's weight may be what that kernel writes."""
    run(fake, f"""
fake.fake_reset()
ok(lib.kc_rms_norm(ctx, at, at, 2, {dim}, 1e-5, at))
assert calls() == ["launch in order"]
""")


@pytest.mark.parametrize("device", [True, False])
def test_a_call_after_a_failed_allocation(fake, device):
    """Growing the metadata arena gives the old one up first. Where the new one cannot be had, the next call has to make one
    of its own size: with the device's memory at its end, or the pinned memory's (the failure is in the second allocation)."""
    run(fake, f"""
ok(attention([(3, 40)]))
fake.fake_fail_above(1 << 16)
if not {device}: fake.fake_fail_host_only(1)
assert attention([(1, 1200)] * 600, heads=2) == L.KC_ERR_OOM
fake.fake_fail_above(2 ** 62)
fake.fake_reset()
ok(attention([(3, 40)]))
assert calls().count("copy") == 1
""")


@pytest.mark.parametrize("out_features", [384, 26700])
def test_rows_beyond_the_chunks_of_one_launch(fake, out_features):
    """Row chunks are the third dimension of a launch's grid, of which there are 65535 at most: more rows are more launches."""
    run(fake, f"""
w = C.c_void_p()
words = C.create_string_buffer({out_features} * 64 // 2 + 256)
ok(lib.kc_qweight_create(ctx, C.cast(words, C.POINTER(C.c_uint32)), words, words, {out_features}, 64, 4, 64, 0, C.byref(w)))
for rows in (1, 700, 40000, 7000000, 17000000):
    fake.fake_reset()
    ok(lib.kc_quantized_matmul(ctx, w, at, rows, at))
    assert calls().count("launch early") >= (1 if rows < 65535 * 192 else 2)
""")


@pytest.mark.parametrize("out_features,in_features,bits,group", [(4096, 14336, 4, 64), (8192, 8192, 4, 64), (3584, 18944, 8, 32), (3584, 14336, 4, 128), (6144, 4096, 4, 64)])
def test_rows_left_over_by_a_large_launch(fake, out_features, in_features, bits, group):
    """Weights that are split along K: a launch of many rows takes the splits in turn and has no limit of 512 rows, the rows
    that the last launch is left with may be too few for that and are launches of 512. All counts are taken, by all calls."""
    run(fake, f"""
w = C.c_void_p()
words = C.create_string_buffer({out_features} * {in_features} * {bits} // 8 + 256)
ok(lib.kc_qweight_create(ctx, C.cast(words, C.POINTER(C.c_uint32)), words, words, {out_features}, {in_features}, {bits}, {group}, 0, C.byref(w)))
in_turn = apart = 0
for rows in [2 ** 20 * k + left for k in (0, 1, 2) for left in (1, 257, 512, 513, 600, 641, 774, 896, 961, 1296, 2000)]:
    fake.fake_reset()
    ok(lib.kc_quantized_matmul(ctx, w, at, rows, at))
    seen = calls().count("launch early")
    in_turn += rows > 512 and seen <= rows // 2 ** 20 + 1
    apart += rows > 2 ** 20 and seen > rows // 2 ** 20 + 1
    rc = lib.kc_quantized_matmul_static(ctx, w, at, rows, at)
    assert rc == L.KC_OK or rc == L.KC_ERR_UNSUPPORTED and rows > 256, (rows, rc, lib.kc_last_error())
assert in_turn and apart, (in_turn, apart)     # both ways, the second one in what a large launch leaves
""")


@pytest.mark.parametrize("segments,old", [
    ([(4, 60, list(range(4)))], [60]),                                  # its own last block holds old and new keys
    ([(4, 64, list(range(5)))], [64]),
    ([(1, 40, [0, 1, 2]), (1, 40, [0, 1, 3])], [40, 40]),               # a shared prefix that neither writes
    ([(16, 0, [7]), (1, 40, [0, 7, 2])], [0, 16]),                      # another sequence writes its second block
    ([(20, 40, [0, 1, 2, 3]), (4, 60, [0, 1, 2, 3])], [40, 32]),        # pieces of one sequence
    ([(10, 40, [5, 1, 2, 5])], [0]),                                    # its own writes come to its first block again
    ([(10, 40, [1, 5, 2, 5])], [16]),
    ([(20, 40, [0, 1, 2, 2])], [32]),                                   # .. and to the one that they begin in
    ([(1, 40, [0, 3, 3])], [16]),
    ([(1, 40, [3, 3, 0])], [40]),                                       # named twice, not written
])
def test_keys_that_a_step_writes_are_not_old(fake, segments, old):
    """Attention loads a sequence's old keys before it waits for the kernel ahead, which writes the new ones: none of them may
    lie in a block that the step writes at another position or for another sequence. Read off the units that are copied."""
    run(fake, f"""
import struct
segments, old = {segments}, {old}
tables = [(C.c_uint32 * len(b))(*b) for _, _, b in segments]
seqs = (L.KcSeqStep * len(segments))(*[L.KcSeqStep(n, off, n, len(b), t) for (n, off, b), t in zip(segments, tables)])
rows = sum(n for n, _, _ in segments)
ok(lib.kc_paged_attention(ctx, kv, 0, at, rows, 4, seqs, len(segments), 0.125, 0.0, 0, at))
fake.fake_copied.restype, size = C.c_void_p, C.c_size_t()
data = C.string_at(fake.fake_copied(C.byref(size)), size.value)
found, row = [], 0
for i, (n, off, _) in enumerate(segments):
    units = [j for j in range(0, len(data) - 31, 16) if data[j: j + 24] == struct.pack("6i", i, row, n, off, 0, 1)]   # sequence, rows, position, chunk 0 alone
    assert len(units) == 1, (i, units)
    found.append(struct.unpack_from("i", data, units[0] + 28)[0])
    row += n
assert found == old, (found, old)
""")


@pytest.mark.parametrize("out_features,in_features,bits,rows,in_turn", [
    (4096, 4096, 4, 384, False), (4096, 4096, 4, 512, True), (4096, 4096, 4, 2048, True), (4096, 14336, 4, 2048, True), (6144, 4096, 4, 2048, True),
    (7000, 28672, 4, 1200, False), (8192, 28672, 4, 1500, False), (1024, 8192, 4, 768, False), (1024, 8192, 4, 2048, True), (2048, 8192, 4, 513, False),
    (2048, 8192, 4, 1024, True)])
def test_many_rows_take_the_faster_way(fake, out_features, in_features, bits, rows, in_turn):
    """One launch with the splits in turn, or launches of 512 rows with a reduction each: on both sides of the rule, where each
    way was measured to be the faster one by a twentieth or more."""
    run(fake, f"""
w = C.c_void_p()
words = C.create_string_buffer({out_features} * {in_features} * {bits} // 8 + 256)
ok(lib.kc_qweight_create(ctx, C.cast(words, C.POINTER(C.c_uint32)), words, words, {out_features}, {in_features}, {bits}, 64, 0, C.byref(w)))
fake.fake_reset()
ok(lib.kc_quantized_matmul(ctx, w, at, {rows}, at))
assert calls().count("launch early") == ({1 if in_turn else 2 * -(-rows // 512)})
""")


@pytest.mark.parametrize("hd,gqa,lens,cap,keys_up_to", [
    # one short sequence; few units of one chunk each; enough of them to fill the SMs; many long sequences (units of whole rows)
    (64, 4, [100], 0, 32), (64, 4, [1001], 0, 0), (64, 4, [3000] * 4, 0, 24), (64, 8, [1400] * 48, 0, 32), (64, 4, [1001], 30, 24), (64, 4, [1400] * 48, 30, 64),
    (128, 4, [100], 0, 32), (128, 4, [1001], 0, 16), (128, 4, [3000] * 4, 0, 32), (128, 4, [1400] * 48, 0, 40), (128, 8, [1001], 30, 32), (128, 4, [1400] * 48, 30, 64),
    (256, 2, [100], 0, 24), (256, 2, [1001], 0, 32), (256, 2, [3000] * 4, 50, 64), (256, 2, [1400] * 48, 0, 64)])
def test_attention_takes_the_faster_kernel(fake, hd, gqa, lens, cap, keys_up_to):
    """A call on its own takes the kernel with a key per thread (768 threads) up to the rows of a unit with which it was
    measured to be the faster one, then that with a row per thread (384)."""
    run(fake, f"""
ok(lib.kc_kv_create(ctx, 1, 8, {hd}, 200, 16, L.KC_BF16, C.byref(kv)))
table = (C.c_uint32 * 200)(*range(200))
lens, gqa = {lens}, {gqa}
for rows in range(1, 64 // gqa + 2):
    seqs = (L.KcSeqStep * len(lens))(*[L.KcSeqStep(rows, n, rows, 200, table) for n in lens])
    ok(lib.kc_paged_attention(ctx, kv, 0, at, rows * len(lens), 8 * gqa, seqs, len(lens), 0.1, {cap}, 0, at))
    assert fake.fake_threads() == (768 if rows * gqa <= {keys_up_to} else 384), rows * gqa
""")


@pytest.mark.parametrize("hidden,heads,kv_heads,hd,rows,qkv,o", [
    (2048, 32, 8, 64, 257, "640:24x4x2", "640:16x4x2"), (2048, 32, 8, 64, 500, "640:24x4x3", "640:16x4x4"),      # splits apart
    (4096, 32, 8, 128, 384, "640:48x3x2", "640:32x4x2"), (4096, 32, 8, 128, 448, "640:144x1x1", "640:128x1x1"),  # .. and in turn
    (3584, 16, 8, 256, 333, "640:64x2x2", "640:28x5x2")])
def test_partials_that_a_consumer_sums(fake, hidden, heads, kv_heads, hd, rows, qkv, o):
    """In a step the kernel behind a linear sums its partials at next to no cost: the linear takes its splits in turn only where
    that is faster by itself. Read off the grids of a layer's first two linears (tiles x splits x chunks of rows, or CTAs)."""
    run(fake, f"""
import dataclasses
import numpy as np
from kiln_b200 import api
from kiln_b200.synth import PRESETS, synth_checkpoint
fake.fake_shapes.restype = C.c_char_p
cfg = dataclasses.replace(PRESETS["tiny-llama"], hidden_size={hidden}, num_attention_heads={heads}, num_key_value_heads={kv_heads}, head_dim={hd},
                          num_hidden_layers=1)
c = api.Context(0)
model = api.CudaModel(c, cfg, synth_checkpoint(cfg, seed=0), max_step_tokens=512, max_step_seqs=1)
pool = api.PagedKv(c, model.kv_spec(32, 16))
p = api._PackedStep(api.StepBatch(np.zeros({rows}, dtype=np.uint32), [api.SeqStep({rows}, 0, 0, list(range(32)))]))
logits, n = C.c_void_p(), C.c_int32()
fake.fake_reset()
ok(L.lib().kc_forward_step(model._h, pool._h, p.ids_p, p.n, p.seq_arr, p.n_seqs, 0, C.byref(logits), C.byref(n)))
grids = [s for s in fake.fake_shapes().decode().split() if s.startswith("640:")]
assert grids[:2] == ["{qkv}", "{o}"], grids
""", first="import torch")   # before the library, whose NCCL is another one


@pytest.mark.parametrize("heads,kv_heads,hd,shape", [(4, 2, 64, "256:3x1x1"), (32, 8, 64, "256:3x1x1"), (48, 8, 64, "256:3x1x1"), (4, 4, 128, "256:3x1x1"), (32, 8, 128, "128:3x3x1"), (16, 8, 256, "128:3x4x1"), (64, 8, 64, "128:3x3x1")])
def test_rope_items_of_a_token(fake, heads, kv_heads, hd, shape):
    """Up to 256 work items of a token are one block's of 256 threads, more are blocks of 128."""
    run(fake, f"""
fake.fake_shapes.restype = C.c_char_p
pool = C.c_void_p()
ok(lib.kc_kv_create(ctx, 1, {kv_heads}, {hd}, 80, 16, L.KC_BF16, C.byref(pool)))
fake.fake_reset()
seqs = (L.KcSeqStep * 1)(L.KcSeqStep(3, 40, 3, 3, table))
ok(lib.kc_rope_kv_write(ctx, pool, 0, at, None, C.cast(at, C.POINTER(C.c_float)), 3, {heads}, 0, seqs, 1, at))
assert fake.fake_shapes().decode().split() == ["{shape}"], fake.fake_shapes()
""")


@pytest.mark.parametrize("heads,kv_heads,hd,offset,rows,threads", [
    (32, 8, 64, 600, 8, 768), (32, 8, 64, 600, 9, 384), (32, 8, 64, 70, 16, 768), (32, 8, 64, 70, 17, 384), (32, 8, 128, 600, 16, 768), (32, 8, 128, 600, 17, 384),
    (16, 8, 256, 600, 32, 768), (16, 8, 256, 600, 33, 384)])
def test_attention_in_a_step_takes_the_faster_kernel(fake, heads, kv_heads, hd, offset, rows, threads):
    """A step's units of up to 64 rows take the kernel with a key per thread (768 threads), 32 at head size 64 and more than
    one chunk."""
    run(fake, f"""
import dataclasses
import numpy as np
from kiln_b200 import api
from kiln_b200.synth import PRESETS, synth_checkpoint
fake.fake_shapes.restype = C.c_char_p
cfg = dataclasses.replace(PRESETS["tiny-llama"], num_attention_heads={heads}, num_key_value_heads={kv_heads}, head_dim={hd}, num_hidden_layers=1)
c = api.Context(0)
model = api.CudaModel(c, cfg, synth_checkpoint(cfg, seed=0), max_step_tokens=64, max_step_seqs=1)
pool = api.PagedKv(c, model.kv_spec(64, 16))
p = api._PackedStep(api.StepBatch(np.zeros({rows}, dtype=np.uint32), [api.SeqStep({rows}, {offset}, 0, list(range(64)))]))
logits, n = C.c_void_p(), C.c_int32()
fake.fake_reset()
ok(L.lib().kc_forward_step(model._h, pool._h, p.ids_p, p.n, p.seq_arr, p.n_seqs, 0, C.byref(logits), C.byref(n)))
threads = [s.split(":")[0] for s in fake.fake_shapes().decode().split()]
assert [t for t in threads if t in ("384", "768")] == ["{threads}"], threads
""", first="import torch")


def test_a_launch_has_the_chunks_that_were_weighed(fake):
    """Rows of 4096 x 14336 that are taken with all splits in turn: four chunks of at most 192 rows are one task for each of 64 teams of two
    SMs. Chunks of fewer rows than the choice was made for would be 80 tasks, two rounds of the 74 teams."""
    run(fake, """
w = C.c_void_p()
src = C.create_string_buffer(4096 * 14336 // 2)
ok(lib.kc_qweight_create(ctx, C.addressof(src), C.addressof(src), C.addressof(src), 4096, 14336, 4, 64, 0, C.byref(w)))
fake.fake_shapes.restype = C.c_char_p
for m in (641, 672, 704, 768):
    fake.fake_reset()
    ok(lib.kc_quantized_matmul(ctx, w, at, m, at))
    assert fake.fake_shapes().decode().split() == ["640:128x1x1"], (m, fake.fake_shapes())
""")


def test_a_weight_loads_without_room_for_what_teams_leave(fake):
    """A wide weight's launches cut its pairs of tiles between teams, which takes a workspace of 44 MB: a weight that fits the device's
    memory without it loads, and its launches have whole pairs."""
    run(fake, """
w = C.c_void_p()
src = C.create_string_buffer(26700 * 2304 // 2 + 256)
fake.fake_fail_above(41 << 20)
ok(lib.kc_qweight_create(ctx, C.addressof(src), C.addressof(src), C.addressof(src), 26700, 2304, 4, 64, 0, C.byref(w)))
fake.fake_fail_above(2 ** 62)
fake.fake_reset()
ok(lib.kc_quantized_matmul(ctx, w, at, 5, at))
assert [c for c in calls() if c != "sync"] == ["launch early"]
""")
