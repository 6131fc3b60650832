"""Nothing outside of a process puts its products on CTA pairs: whole steps on that kernel were seen to stop. Asks the kernel library which
form it would run; no GPU, nothing is launched."""
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
ASK = """
import sys
sys.path.insert(0, {path!r})
import torch
torch.cuda.is_available = lambda: True
from llmengine.ops import CudaOps
print([CudaOps().gemm_form(m, n, k, s) for m, n, k, s in ((2048, 16384, 3072, True), (2048, 3072, 8192, False), (300, 25617, 192, False))])
"""


@pytest.mark.parametrize("value", ["on", "auto", "off"])
def test_the_environment_does_not_choose_the_pair_kernel(value):
    code = ASK.format(path=os.path.join(ROOT, "llm-inference-engine-v6_b200"))
    r = subprocess.run([sys.executable, "-c", code], env=dict(os.environ, LLMENGINE_CTA_PAIRS=value), stdout=subprocess.PIPE, stderr=subprocess.PIPE, text=True)
    assert r.returncode == 0, r.stderr
    assert "persistent" in r.stdout and "CTA pairs" not in r.stdout
