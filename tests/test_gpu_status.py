"""What a bounded wait that gave up does to pipelined launches. No wait gives up here: the test writes the context's
status word from the host, in a process of its own, and the kernels read it."""
import ctypes as C
import os
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parent.parent
CODE = 0x201


def test_a_failed_launch_stays_failed_and_fails_no_other(tmp_path):
    shim = tmp_path / "status_word.so"
    subprocess.run(["g++", "-shared", "-fPIC", "-I/usr/local/cuda/include", "-o", str(shim), str(ROOT / "tests" / "status_word.cpp"), "-ldl"], check=True)
    r = subprocess.run([sys.executable, __file__], cwd=ROOT, env={**os.environ, "LD_PRELOAD": str(shim), "PYTHONPATH": str(ROOT)},
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "STATUS CHECK PASSED" in r.stdout


def main():
    import torch
    from kiln_b200 import _lib as L
    from kiln_b200 import api
    from kiln_b200.synth import PRESETS, synth_checkpoint

    ctx = api.Context(0)
    shim = C.CDLL(None)
    shim.status_word.restype = C.c_void_p
    word = C.c_uint32.from_address(shim.status_word())
    stream = torch.cuda.ExternalStream(ctx.stream)
    cfg = PRESETS["tiny-llama"]
    models = [api.CudaModel(ctx, cfg, synth_checkpoint(cfg, seed=s), max_step_tokens=64, max_step_seqs=4) for s in (0, 1)]
    pools = [api.PagedKv(ctx, m.kv_spec(8, 16)) for m in models]
    at = [0, 0]

    def launch(i, feed=-1):
        t = models[i].decode_launch(api.StepBatch([5], [api.SeqStep(1, at[i], 1, [1, 2])]), pools[i], [feed])
        at[i] += 1
        return t

    def timeout(call, *args):
        try:
            call(*args)
        except api.KcError as e:
            assert e.code == L.KC_ERR_TIMEOUT and f"0x{CODE:x}" in e.message, e
        else:
            raise AssertionError("the call returned")

    def collect(i, t):
        return models[i].decode_collect(t, 1)

    row = lambda i: api.StepBatch([5], [api.SeqStep(1, 0, 1, [3])])
    between = [ctx.sync, lambda: models[0].verify_step(row(0), pools[0]), lambda: models[0].draft_chain(pools[0], 5, 0, [3], 2),
               lambda: models[1].verify_step(row(1), pools[1])]
    for call in between:                  # another call reports the code and clears the word before the launch is collected
        good = launch(0)
        stream.synchronize()
        word.value = CODE
        bad = launch(0, 0)
        timeout(call)
        assert word.value == 0
        assert len(collect(0, good)) == 1
        timeout(collect, 0, bad)
    ctx.sync()
    a = launch(0)                         # two models on one context: the failure is the second one's
    stream.synchronize()
    word.value = CODE
    b = launch(1)
    stream.synchronize()
    assert len(collect(0, a)) == 1
    timeout(collect, 1, b)
    ctx.sync()
    word.value = CODE                     # a launch that is already behind a failed one has failed as well
    a = launch(0)
    b = launch(0, 0)
    stream.synchronize()
    timeout(collect, 0, a)
    timeout(collect, 0, b)
    ctx.sync()
    assert len(collect(0, launch(0))) == 1 and ctx.device_status() == 0
    print("STATUS CHECK PASSED")


if __name__ == "__main__":
    main()
