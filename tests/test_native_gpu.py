"""The native host path of the device calls against the Python one: same bits out, and a call that it does not serve (another
type, a wrong shape, a CPU tensor) falls through to the wrapper's own conversion or error."""
import numpy as np
import pytest
import torch

import quactlize_b200 as qb
from quactlize_b200 import _lib, synth

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
K = 1024


class _Absent:
    def __getattr__(self, name):
        return lambda *a: None


def _cuda(a):
    return torch.from_numpy(np.ascontiguousarray(a)).to(DEV)


def _calls(qtype, n, m):
    """name -> a call with its arguments made"""
    g = qb.kquant_geometry(qtype)
    blocks = synth.kquant_blocks(qtype, n * K // 256, seed=qtype)
    b, x = _cuda(blocks), _cuda(synth.activations(m, K, seed=2))
    low, high, units = (t.to(DEV) for t in qb.gguf_prepare_fully_quantized_dense(torch.from_numpy(blocks), n, K, qtype))
    sf = tuple(t.to(DEV) for t in qb.gguf_prepare_gemv(torch.from_numpy(blocks), n, K, qtype))
    lo, sc, ze = (_cuda(t) for t in synth.group_planes(2, n, K, 4, 64, seed=3))
    off = torch.tensor([0, m - 1, m], dtype=torch.int32, device=DEV)
    one = x[:1].contiguous()
    return {
        "dense": lambda: qb.gguf_vecdot_dense(b, one, n, K, qtype),
        "rows": lambda: qb.gguf_vecdot_rows(b, x, n, K, qtype),
        "generic": lambda: qb.gguf_vecdot_rows(b, x, n, K, qtype, True),
        "dense2": lambda: torch.cat(qb.gguf_vecdot_dense2(b, b, one, n, n, K, qtype)),
        "dequantize": lambda: qb.gguf_dequantize(b, qtype),
        "bc": lambda: qb.gguf_gemv_bc(one, low, high, units, qtype),
        "scale_first": lambda: qb.gguf_gemv_scale_first(x, *sf, qtype),
        "moe": lambda: qb.gguf_vecdot_moe(b.view(2, -1, b.shape[1]), x, off, qtype),
        "plane": lambda: qb.gemv_plane(x, lo[:1], None, sc[:1], ze[:1], 4, 0, 64),
        "plane_no_zero": lambda: qb.gemv_plane(x, lo[:1], None, sc[:1], None, 4, 0, 64, code_offset=-8),
        "plane_two": lambda: qb.gemv_plane(x, sf[0], sf[1] if g.hi_bits else None, sf[2], sf[3], g.lo_bits, g.hi_bits, g.group_size),
        "plane_moe": lambda: qb.gemv_plane(x.bfloat16(), lo, None, sc, ze, 4, 0, 64, row_offsets=off, max_rows=m),
        "gemm": lambda: qb.gemm_plane(x, lo[:1], None, sc[:1], ze[:1], 4, 0, 64),
        "gemm_moe": lambda: qb.gemm_plane(x.bfloat16(), lo, None, sc, ze, 4, 0, 64, row_offsets=off),
        "fq": lambda: qb.gguf_dense_fully_quantized(x, low, high, units, qtype),
    }


@pytest.mark.parametrize("n,m", [(256, 2), (512, 5)])
@pytest.mark.parametrize("qt", [10, 12, 14])
def test_native_path_gives_the_python_path_s_bits(monkeypatch, qt, n, m):
    calls = _calls(qt, n, m)
    native = {name: f() for name, f in calls.items()}
    torch.cuda.synchronize()
    monkeypatch.setattr(qb, "_native", _Absent())
    for name, f in calls.items():
        want = f()
        assert native[name].dtype == want.dtype and native[name].shape == want.shape, name
        assert torch.equal(native[name].view(torch.uint8), want.view(torch.uint8)), name
    assert _lib.lib().quactlize_b200_device_wait_status() == 0


def test_calls_it_does_not_serve_fall_through():
    n = 256
    blocks = torch.from_numpy(synth.kquant_blocks(12, n * K // 256, seed=1))
    b = blocks.to(DEV)
    x = _cuda(synth.activations(1, K, seed=2))
    want = qb.gguf_vecdot_dense(b, x, n, K, 12)
    assert torch.equal(qb.gguf_vecdot_dense(b, x.float(), n, K, 12), want)                       # converted
    wide = torch.empty((1, 2 * K), dtype=torch.float16, device=DEV)
    wide[:, ::2] = x
    assert torch.equal(qb.gguf_vecdot_dense(b, wide[:, ::2], n, K, 12), want)                    # made contiguous
    assert torch.equal(qb.gguf_vecdot_dense(b, x, np.int64(n), K, qb.QuantType.Q4_K), want)      # integer-like arguments
    with torch.cuda.stream(torch.cuda.Stream()) as _:
        side = qb.gguf_vecdot_dense(b, x, n, K, 12)                                              # another stream
    torch.cuda.synchronize()
    assert torch.equal(side, want)
    assert torch.equal(qb.gguf_vecdot_dense(blocks, x.cpu(), n, K, 12), want.cpu())              # host tensors
    for bad in (lambda: qb.gguf_vecdot_dense(b, x, n + 1, K, 12), lambda: qb.gguf_vecdot_dense(b, x, n, K, 7),
                lambda: qb.gguf_vecdot_dense(b, x.cpu(), n, K, 12), lambda: qb.gguf_vecdot_dense(b.float(), x, n, K, 12),
                lambda: qb.gguf_vecdot_rows(b, x[:, :-1], n, K, 12), lambda: qb.gguf_dequantize(b[:, :-1], 12)):
        with pytest.raises(RuntimeError):
            bad()
