"""Errors raised by the operators' C++ side arrive as Python exceptions (no GPU: fake tensors reach the checks, nothing runs)."""
import subprocess
import sys

from conftest import ROOT

CALLS = """
import torch
from torch._subclasses.fake_tensor import FakeTensorMode
import fastalgebraictransformer_b200 as fat
with FakeTensorMode():
    q, slopes = torch.empty(1, 2, 64, 64, device="cuda"), torch.empty(2, device="cuda")
    assert fat.rational_attention(q, q, q, slopes, 0.125).shape == q.shape
    for shape, text in (((1, 1, 64), "must be [B, T]"), ((1, 65), "covers 65 tokens, the sequence has 64")):
        try:
            fat.rational_attention(q, q, q, slopes, 0.125, key_mask=torch.ones(shape, device="cuda"))
        except ValueError as e:
            assert text in str(e), e
        else:
            raise SystemExit("accepted")
"""


def test_an_error_text_with_numbers_reaches_python():
    r = subprocess.run([sys.executable, "-c", CALLS], cwd=ROOT, capture_output=True, text=True)      # (a process of its own: this once crashed)
    assert r.returncode == 0, r.stderr[-2000:]
