"""The threaded, word-wide host producers against the oracle at sizes that are dealt to several threads: row counts off the
row tile, an odd number of rows per expert, one row."""
import os
import shutil
import subprocess

import numpy as np
import pytest
import torch

import quactlize_b200 as qb
from oracle import kquant as kq
from quactlize_b200 import synth


def _bits(t):
    return np.asarray(t).view(np.uint16) if np.asarray(t).dtype == np.float16 else np.asarray(t)


@pytest.mark.parametrize("n,k,experts", [(1, 512, 1), (33, 512, 3), (1031, 4096, 1), (1200, 3072, 2)])
def test_producers_match_the_oracle(qtype, n, k, experts):
    blocks = synth.kquant_blocks(qtype, experts * n * k // 256, seed=qtype + n)
    tb = torch.from_numpy(blocks)
    want = kq.prepare_gemv(blocks, experts * n, k, qtype)
    got = qb.gguf_prepare_gemv(tb.view(experts, -1, blocks.shape[1]), n, k, qtype)
    for g, w in zip(got[:2], want[:2]):                                      # planes: experts are further rows
        assert np.array_equal(g.numpy().reshape(-1), np.asarray(w).reshape(-1))
    for g, w in zip(got[2:], want[2:]):                                      # fp16 planes [1, k/gs, E*n] against [E, k/gs, n]
        w = np.asarray(w).reshape(-1, experts, n).transpose(1, 0, 2)
        assert np.array_equal(_bits(g.numpy()), _bits(np.ascontiguousarray(w)))
    units = qb.gguf_pack_units(tb, n, k, qtype, experts).numpy()
    per = n * k // 256
    for e in range(experts):
        assert np.array_equal(units[e], np.asarray(kq.pack_units(blocks[e * per:(e + 1) * per], n, k, qtype)[0]))


@pytest.mark.parametrize("flags", [[], ["-U__SSE2__"]])
def test_plain_squeezer_equals_the_vector_one(tmp_path, flags):
    """The producers build on hosts without SSE2 (the header then has the plain form only) and write the same bytes."""
    if shutil.which("g++") is None:
        pytest.skip("no C++ compiler")
    here = os.path.dirname(os.path.abspath(__file__))
    exe = tmp_path / "probe"
    subprocess.run(["g++", "-std=c++17", "-O1", *flags, "-I", os.path.join(os.path.dirname(here), "quactlize_b200", "csrc"),
                    os.path.join(here, "host_squeeze_probe.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
