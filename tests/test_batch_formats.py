"""The per-format operand builders of the batch kernel (gguf_jax_b200/csrc/batch_formats.cuh) on the CPU: scaled codes, both planes,
offsets and the order of the activations reproduce the decoded weights bit for bit.  They are compared with the block decoders over
all code values and scales that random bytes give."""
import os
import subprocess

import numpy as np
import pytest
from gguf.constants import GGMLQuantizationType as QT

from gguf_jax_b200 import synth
from oracle import oracle as O
from tests.test_tile_formats import kernel_table

SRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "native", "batch_formats_check.cpp")
BATCH_QTYPES = [QT.Q2_K, QT.Q3_K, QT.Q4_K, QT.Q5_K, QT.Q6_K, QT.IQ4_XS, QT.IQ2_XXS, QT.IQ2_XS, QT.IQ2_S, QT.IQ3_XXS, QT.IQ3_S, QT.IQ1_S,
                QT.IQ1_M, QT.TQ1_0, QT.TQ2_0]


@pytest.fixture(scope="module")
def checker(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("native") / "batch_formats_check")
    cxx = "/usr/bin/g++" if os.path.exists("/usr/bin/g++") else "g++"
    subprocess.run([cxx, "-O1", "-std=c++17", "-ffp-contract=off", "-o", exe, SRC], check=True, capture_output=True)
    return exe


@pytest.mark.parametrize("qtype", BATCH_QTYPES, ids=lambda t: t.name)
def test_scaled_operands_reproduce_the_decoded_weights(qtype, checker, tmp_path):
    n_blocks = 400
    blocks = synth.random_blocks(qtype, n_blocks, seed=int(qtype))
    dense = O.c_dequantize(blocks, qtype).astype(np.float32)
    (tmp_path / "b.bin").write_bytes(blocks.tobytes())
    (tmp_path / "d.bin").write_bytes(dense.tobytes())
    (tmp_path / "t.bin").write_bytes(kernel_table(qtype))
    r = subprocess.run([checker, str(int(qtype)), str(tmp_path / "b.bin"), str(tmp_path / "d.bin"), str(tmp_path / "t.bin"), str(n_blocks)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "0 mismatches" in r.stdout
