"""Raw-block kernel for several activation rows (csrc/qb_gemv_kqrows.cu) at the edges of its tiles, passes and alignments.

Its operands are exact (fp16 activations, sub-scale x code products of at most 11 bits), so what is left is the fp32
accumulation of the tensor cores: at most a few units of 2^-23 of the sum of the terms' sizes, which for K normal terms
is about sqrt(K)/3 times the largest output: 2e-5 of the largest output at K = 16384.
"""
import numpy as np
import pytest
import torch

import quactlize_b200 as qb
from oracle import kquant as kq
from quactlize_b200 import _lib, synth

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
QTYPES = (10, 11, 12, 13, 14)


def _cuda(a):
    return torch.from_numpy(np.ascontiguousarray(a)).to(DEV)


# (rows, n, k): one tile and its edges, every split of the warps and of K (passes, clusters), K whose rows end off a
# 16-byte boundary, activation rows at and beyond one group of eight
@pytest.mark.parametrize("m,n,k", [(2, 16, 256), (3, 17, 512), (8, 15, 1280), (5, 130, 2304), (9, 48, 1024), (4, 2500, 1024),
                                   (7, 333, 4096), (2, 1000, 4352), (8, 600, 14336), (6, 5000, 5376), (1, 77, 768), (3, 40, 33024)])
@pytest.mark.parametrize("qt", QTYPES)
def test_rows(qt, m, n, k):
    blocks = synth.kquant_blocks(qt, n * k // 256, seed=qt + m)
    x = synth.activations(m, k, seed=n)
    out = qb.gguf_vecdot_rows(_cuda(blocks), _cuda(x), n, k, qt).cpu().numpy()
    ref = np.concatenate([kq.vecdot_dense(blocks, x[i:i + 1], n, k, qt).reshape(1, n) for i in range(m)])
    fp16_sums = m <= 2 and (qt in (12, 13) or k // 256 % 8 == 0)     # the one-row kernels
    assert kq.max_rel(out, ref) < (4e-3 if fp16_sums else 2e-5)


@pytest.mark.parametrize("qt,m,n,k", [(12, 2, 500, 8192), (12, 3, 200, 14336), (12, 2, 100, 4352),
                                      (13, 2, 200, 14336), (14, 3, 100, 14336), (10, 3, 100, 10240), (11, 2, 60, 12288)])
def test_sums_are_fp32_on_deep_rows(qt, m, n, k):
    blocks = synth.kquant_blocks(qt, n * k // 256, seed=m)
    x = synth.activations(m, k, seed=n)
    out = qb.gguf_vecdot_rows(_cuda(blocks), _cuda(x), n, k, qt).cpu().numpy()
    assert kq.max_rel(out, np.concatenate([kq.vecdot_dense(blocks, x[i:i + 1], n, k, qt).reshape(1, n) for i in range(m)])) < 2e-5


# K over clusters of two CTAs, each in two passes: many tiles of deep rows
@pytest.mark.parametrize("qt,m,n,k", [(12, 2, 4736, 14336), (13, 5, 4736, 9216), (14, 3, 7104, 8448)])
def test_rows_deep_and_wide(qt, m, n, k):
    blocks = synth.kquant_blocks(qt, n * k // 256, seed=m)
    x = synth.activations(m, k, seed=n)
    out = qb.gguf_vecdot_rows(_cuda(blocks), _cuda(x), n, k, qt).cpu().numpy()
    rows = np.random.default_rng(k).choice(n, 200, replace=False)
    sub = np.ascontiguousarray(blocks.reshape(n, k // 256, -1)[rows]).reshape(200 * k // 256, -1)
    want = x.astype(np.float64) @ kq.dequantize_f32(sub, qt).reshape(200, k).T
    assert kq.max_rel(out[:, rows], want) < 2e-5


@pytest.mark.parametrize("k", [2304, 4352, 13568])
@pytest.mark.parametrize("qt", QTYPES)
def test_error_against_64_bits(qt, k):
    """Eight rows whose blocks start off a 16-byte boundary where the format allows it.  A sum of thousands of fp32 terms in chains of
    at most eight tensor-core steps and a pairwise tail: two and a half units of 2^-24 of the result's 2-norm."""
    m, n = 8, 256
    blocks = synth.kquant_blocks(qt, n * k // 256, seed=qt + k)
    x = np.random.default_rng(k).standard_normal((m, k)).astype(np.float16)
    want = x.astype(np.float64) @ kq.dequantize_f32(blocks, qt).reshape(n, k).T
    got = qb.gguf_vecdot_rows(_cuda(blocks), _cuda(x), n, k, qt).cpu().numpy()
    assert np.linalg.norm(got - want) < 2.5 * 2.0**-24 * np.linalg.norm(want)


@pytest.mark.parametrize("counts", [[0, 0, 1, 0], [3, 0, 17, 8, 1], [1] * 16, [0, 9, 0, 0, 0, 0, 2]])
@pytest.mark.parametrize("n,k", [(70, 768), (300, 2304), (40, 8448)])
@pytest.mark.parametrize("qt", QTYPES)
def test_moe(qt, n, k, counts):
    e, rows = len(counts), sum(counts)
    blocks = synth.kquant_blocks(qt, e * n * k // 256, seed=qt).reshape(e, n * k // 256, -1)
    x = synth.activations(rows, k, seed=3)
    off = np.concatenate([[0], np.cumsum(counts)]).astype(np.int32)
    out = qb.gguf_vecdot_moe(_cuda(blocks), _cuda(x), _cuda(off), qt).cpu().numpy()
    assert kq.max_rel(out, kq.vecdot_moe(blocks, x, off, n, k, qt)) < 2e-5


@pytest.mark.parametrize("qt", QTYPES)
def test_blocks_off_a_16_byte_boundary(qt):
    """A view into a larger buffer: 16-byte formats need the plain kernel there, the others start mid-unit."""
    m, n, k = 3, 40, 1024
    blocks = synth.kquant_blocks(qt, n * k // 256, seed=qt)
    x = synth.activations(m, k, seed=1)
    want = np.concatenate([kq.vecdot_dense(blocks, x[i:i + 1], n, k, qt).reshape(1, n) for i in range(m)])
    for shift in (2, 4, 8):
        buf = torch.zeros(blocks.size + 64, dtype=torch.uint8, device=DEV)
        view = buf[shift:shift + blocks.size].view(blocks.shape)
        view.copy_(_cuda(blocks))
        out = qb.gguf_vecdot_rows(view, _cuda(x), n, k, qt).cpu().numpy()
        assert kq.max_rel(out, want) < 2e-5, shift


@pytest.mark.parametrize("e,n,k,rows", [(64, 1184, 256, 64), (1500, 33, 512, 40)])
@pytest.mark.parametrize("qt", [10, 12])
def test_moe_takes_one_kernel_whoever_asks(qt, e, n, k, rows):
    """At most two rows per expert and many tiles, or many experts: the native call, the converting one and the C ABI agree to the
    last bit, and sums are fp32."""
    blocks = synth.kquant_blocks(qt, e * n * k // 256, seed=qt).reshape(e, n * k // 256, -1)
    x = synth.activations(rows, k, seed=3)
    off = np.concatenate([[0], np.cumsum(np.random.default_rng(e).permutation([1] * rows + [0] * (e - rows)))]).astype(np.int32)
    b, xx, o = _cuda(blocks), _cuda(x), _cuda(off)
    native = qb.gguf_vecdot_moe(b, xx, o, qt)
    assert torch.equal(native, qb.gguf_vecdot_moe(b, xx.float(), o, qt))
    out = torch.empty((rows, n), device=DEV)
    rc = _lib.lib().quactlize_b200_vecdot_moe_dev_v1(b.data_ptr(), b.shape[2], xx.data_ptr(), o.data_ptr(), out.data_ptr(), n, k // 256, e, rows, 1, qt,
                                                     torch.cuda.current_stream().cuda_stream)
    assert rc == 0 and torch.equal(native, out)
    assert kq.max_rel(native.cpu().numpy(), kq.vecdot_moe(blocks, x, off, n, k, qt)) < 2e-5


@pytest.mark.parametrize("qt,m,n,k", [(12, 4, 600, 14336), (14, 8, 300, 4096)])
def test_captured_launch(qt, m, n, k):
    """A cluster launch and a plain one, captured with their plan already made and replayed on other activations."""
    blocks = synth.kquant_blocks(qt, n * k // 256, seed=qt)
    b, x = _cuda(blocks), _cuda(synth.activations(m, k, seed=1))
    qb.gguf_vecdot_rows(b, x, n, k, qt)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = qb.gguf_vecdot_rows(b, x, n, k, qt)
    for seed in (2, 3):
        x.copy_(_cuda(synth.activations(m, k, seed=seed)))
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, qb.gguf_vecdot_rows(b, x, n, k, qt))


def test_moe_refuses_bad_offsets():
    """Offsets that do not describe the rows raise, whatever was enqueued meanwhile, and the next call is right."""
    e, n, k = 3, 64, 1024
    blocks = synth.kquant_blocks(12, e * n * k // 256, seed=5).reshape(e, n * k // 256, -1)
    x = synth.activations(6, k, seed=3)
    b, xx = _cuda(blocks), _cuda(x)
    for bad in ([0, 2, 4, 5], [1, 2, 4, 6], [0, 5, 2, 6], [0, -3, 4, 6], [0, 2, 400000, 6], [0, 2, 6]):
        with pytest.raises(RuntimeError):
            qb.gguf_vecdot_moe(b, xx, torch.tensor(bad, dtype=torch.int32, device=DEV), 12)
    off = np.array([0, 0, 5, 6], dtype=np.int32)
    out = qb.gguf_vecdot_moe(b, xx, _cuda(off), 12).cpu().numpy()
    assert kq.max_rel(out, kq.vecdot_moe(blocks, x, off, n, k, 12)) < 2e-5


@pytest.mark.parametrize("off,used", [([0, 6, 0, 6, 0], [6, 0, 0, 0]), ([2, 1, 5, 3, 9], [0, 3, 0, 1]), ([-4, 6, -1, 2, 7], [6, 0, 0, 0])])
def test_unchecked_offsets_are_settled(off, used):
    """The entry that may be enqueued before its offsets are checked: offsets are clamped to the rows and never fall, so a row
    belongs to one expert and the rows of the others are left alone."""
    e, n, k, rows = 4, 40, 768, 6
    blocks = synth.kquant_blocks(12, e * n * k // 256, seed=8).reshape(e, n * k // 256, -1)
    x = synth.activations(rows, k, seed=4)
    b, xx, out = _cuda(blocks), _cuda(x), torch.full((rows, n), 77.0, device=DEV)
    o = torch.tensor(off, dtype=torch.int32, device=DEV)
    rc = _lib.lib().quactlize_b200_vecdot_moe_clamped_dev_v1(b.data_ptr(), b.shape[2], xx.data_ptr(), o.data_ptr(), out.data_ptr(), n, k // 256,
                                                             e, rows, 12, torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    first = min(max(off[0], 0), rows)
    settled = np.concatenate([[0], np.cumsum(used)]).astype(np.int32)
    want = np.full((rows, n), 77.0, dtype=np.float32)
    want[first:first + settled[-1]] = kq.vecdot_moe(blocks, x[first:first + settled[-1]], settled, n, k, 12)
    assert kq.max_rel(out.cpu().numpy(), want) < 2e-5
