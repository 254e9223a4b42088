"""The host codec on every half and on every code under scales of all kinds, against the oracle's restatement."""
import subprocess
import sys

import numpy as np
import pytest
import torch

import fp6_marlin_b200 as fm
from conftest import ROOT
from oracle import formats as F


def _codes(stream, n, k):
    b = stream.numpy().view(np.uint8).reshape(n, k // 4, 3).astype(np.uint32)
    word = (b[..., 0] << 16) | (b[..., 1] << 8) | b[..., 2]
    return np.stack([(word >> s) & 63 for s in (18, 12, 6, 0)], axis=-1).reshape(n, k).astype(np.uint8)


def test_quantize_codes_every_half_in_range_and_refuses_the_others():
    vals = torch.arange(0, 1 << 16, dtype=torch.int32).to(torch.int16).view(torch.float16)
    mag = vals.abs().float()
    ok = (mag == 0) | ((mag >= 0.0625) & (mag <= 28.0))
    x = torch.zeros(256 * 256, dtype=torch.float16)
    x[: int(ok.sum())] = vals[ok]
    codes = _codes(fm.quantize(x.view(256, 256)), 256, 256).reshape(-1)
    assert np.array_equal(codes, fm.encode_fp6(x).numpy())
    for bad in vals[~ok][:: 997].tolist() + [float("nan"), float("inf"), 28.02, 0.0624]:
        y = x.clone()
        y[-1] = bad
        with pytest.raises(ValueError):
            fm.quantize(y.view(256, 256))


def test_dequantize_every_code_under_every_kind_of_scale():
    n, k = 256, 256
    scales = torch.from_numpy(np.linspace(0, 0x7FFF, n).astype(np.int16)).view(torch.float16).clone()    # subnormal .. infinity, NaN
    scales[::7] *= -1
    rng = np.random.default_rng(0)
    stream = torch.from_numpy(rng.integers(0, 256, n * k * 3 // 4, dtype=np.uint8).view(np.int32).reshape(n, k * 3 // 16).copy())
    value = fm.decode_fp6(torch.from_numpy(_codes(stream, n, k)))
    expect = (value.float() * scales.float()[:, None]).half()
    got = fm.dequantize(stream, scales)
    assert torch.equal(got.isnan(), expect.isnan())
    assert torch.equal(got.nan_to_num(7.0), expect.nan_to_num(7.0))


@pytest.mark.parametrize("n,k", [(256, 256), (512, 768)])
def test_prepacking_places_every_code(n, k):
    """Unpacking the reference layout gives the codes of the stream back."""
    rng = np.random.default_rng(n)
    stream = torch.from_numpy(rng.integers(0, 256, n * k * 3 // 4, dtype=np.uint8).view(np.int32).reshape(n, k * 3 // 16).copy())
    packed = fm.prepacking(stream)
    B, s = fm.repack_from_reference(packed, torch.ones(n, dtype=torch.float16), k, n, n)
    _, c6, _, _ = fm.unpack_b200(B, s, k, n, n, -1)
    assert np.array_equal(c6.numpy(), _codes(stream, n, k).T)


def test_no_thread_and_no_memory():
    """Without room for the stack of a thread (or for the codes that re-tiling keeps) the host functions run on the calling thread
    (or report it): no exception leaves a C entry, which would end the process."""
    program = """
import resource, torch
import fp6_marlin_b200 as fm
from fp6_marlin_b200 import _lib

k, n = 256, 512
torch.manual_seed(0)
x, s = fm.fake_quantize_fp6(torch.randn((k, n)).half())
B, ref = torch.randint(-2**31, 2**31, (k * n * 3 // 16,)).int(), torch.rand(n).half()
q4, s4 = torch.randint(0, 16, (k, n), dtype=torch.uint8), torch.rand((k // 128, n)).half()
def work():
    codes = fm.quantize(x)
    stream = codes.view(n, k * 3 // 16)
    return [codes, fm.prepacking(stream), fm.dequantize(stream, s), fm.encode_fp6(x), *fm.pack_b200(q4, None, s4, None, k, n, -1, 128),
            *fm.repack_from_reference(B, ref, k, n, n)]
expect = work()
big_k, big_n = 16384, 8192
big = torch.zeros(big_k * big_n // 8, dtype=torch.int32)
out, out_s = torch.zeros(fm.b200_sizes(big_k, big_n)[0], dtype=torch.int32), torch.zeros(big_n).half()
pages = int(open('/proc/self/statm').read().split()[0])
resource.setrlimit(resource.RLIMIT_AS, (pages * resource.getpagesize() + (4 << 20),) * 2)
assert all(torch.equal(a, b) for a, b in zip(work(), expect))
rc = _lib.lib.fp6m_repack_from_reference(big.data_ptr(), out_s.data_ptr(), big_k, big_n, -1, out.data_ptr(), out_s.data_ptr())
assert rc == _lib.ERR_NO_MEMORY, rc
print("ok")
"""
    run = subprocess.run([sys.executable, "-c", program], cwd=ROOT, capture_output=True, text=True, timeout=120)
    assert run.returncode == 0 and run.stdout.strip() == "ok", run.stdout + run.stderr
