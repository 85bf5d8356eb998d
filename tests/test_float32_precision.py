"""The float32 training step under every way a program has of allowing TF32 in torch's products.  The setting is the process's
and cannot be unset, so each runs in a process of its own."""

import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SETTINGS = [
    ("pass", True),
    ("torch.set_float32_matmul_precision('highest')", True),
    ("torch.backends.cuda.matmul.allow_tf32 = False", True),
    ("torch.backends.cuda.matmul.fp32_precision = 'ieee'", True),
    ("torch.backends.fp32_precision = 'tf32'; torch.backends.cuda.matmul.fp32_precision = 'ieee'", True),
    ("torch.set_float32_matmul_precision('high')", False),
    ("torch.backends.cuda.matmul.allow_tf32 = True", False),
    ("torch.backends.cuda.matmul.fp32_precision = 'tf32'", False),
    ("torch.backends.fp32_precision = 'tf32'", False),
]

STEP = """
import torch
from flash_moe_b200 import FlashMoE, FlashMoEConfig
torch.manual_seed(0)
with torch.device("cuda"):
    layer = FlashMoE(FlashMoEConfig(256, 512, "silu", 1024, 8, True)).train()
    x, dy = torch.randn(2, 50, 256), torch.randn(2, 50, 256)
y, _ = layer(x)
y.backward(dy)
got = layer.up_proj.weight.grad.double()
X, wg, wu, wd = (t.detach().double().reshape(-1, t.shape[-1]) for t in (x, layer.gate_proj.weight, layer.up_proj.weight, layer.down_proj.weight))
db = dy.double().reshape(-1, 256) @ wd * torch.nn.functional.silu(X @ wg.t())
want = db.t() @ X
error = float((got - want).norm() / want.norm())
"""


def run(code):
    done = subprocess.run([sys.executable, "-c", "import torch\n" + code], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert done.returncode == 0, done.stderr[-2000:]


def test_own_float32_products_follow_both_interfaces():
    """Own products, which do not round, where TF32 is off; torch's where it is on.  Asking leaves the legacy interface usable."""
    procs = [(s, own, subprocess.Popen([sys.executable, "-c", f"import torch\n{s}\nfrom flash_moe_b200.modules.training import "
                                        "_own_float32_products as f\nprint(f(500, 512, 768), f(5000, 512, 768))"],
                                       cwd=ROOT, stdout=subprocess.PIPE, stderr=subprocess.PIPE, text=True)) for s, own in SETTINGS]
    for setting, own, p in procs:
        out, err = p.communicate(timeout=300)
        assert out.split() == [str(own), "False"], (setting, out, err[-500:])
    run("from flash_moe_b200.modules.training import _own_float32_products as f\nf(1, 1, 1)\n"
        "torch.backends.cuda.matmul.allow_tf32 = True\nassert torch.backends.cuda.matmul.allow_tf32 and not f(1, 1, 1)")


@pytest.mark.gpu
@pytest.mark.parametrize("setting,own", [SETTINGS[0], SETTINGS[5], SETTINGS[7], SETTINGS[8]])
def test_float32_step_runs_under_both_interfaces(setting, own):
    """float32: three products in a row, each about sqrt(256) roundings of 2^-24 in its sums, and __expf's 2^-21; TF32 rounds the
    two operands of each by up to 2^-11."""
    run(f"{setting}\n{STEP}\nassert error < {3 * 16 * 2.0**-24 + 2.0**-21 if own else 6 * 2.0**-11}, error")
