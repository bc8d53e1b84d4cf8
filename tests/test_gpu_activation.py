"""The gated activation that the GEMM's epilogue and the element-wise kernel share, over every bf16 gate."""
import ctypes as C
import subprocess
from pathlib import Path

import pytest
import torch

from kiln_b200 import build

ROOT = Path(__file__).resolve().parent.parent

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    so = tmp_path_factory.mktemp("activation") / "check.so"
    subprocess.run([build._nvcc(), *build.NVCC_FLAGS, "-I", str(build.CSRC), "-shared", "-o", str(so), str(ROOT / "tests" / "activation_check.cu")], check=True)
    f = C.CDLL(str(so)).run_check
    f.argtypes = [C.c_int, C.c_void_p, C.c_int, C.c_void_p]
    return f


@pytest.mark.parametrize("gelu", [False, True])
def test_every_gate_has_the_bits_of_the_definition(ctx, check, gelu):
    """silu by a reciprocal without a division's branches, tanh by a polynomial and an exponential: after the rounding to bf16 no gate tells them
    from fp32 division and tanhf, subnormal results, infinities and NaN among them."""
    ups = torch.tensor([1.0, -3.140625, 2.0 ** -20, 2.0 ** 100, -0.0], dtype=torch.bfloat16).view(torch.int16).cuda()
    out = torch.tensor([0, 0, 0x7FFFFFFF], dtype=torch.int32, device="cuda")
    assert check(int(gelu), ups.data_ptr(), ups.numel(), out.data_ptr()) == 0
    one, pair, first = out.tolist()
    assert (one, pair) == (0, 0), f"first at gate bits {first:#06x}"
