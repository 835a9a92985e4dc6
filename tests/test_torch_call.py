"""The extension that takes ordinary calls straight to the C-ABI: same results as the ctypes marshalling
(which `debug=True` still uses), and anything out of the ordinary is declined, so that the Python layer's own
checks and exceptions apply."""
import ctypes
import subprocess
import threading
import time

import pytest
import torch

import kermac_b200 as kermac
from kermac_b200 import _native
from test_grad_split_gpu import full_device


def test_declines_what_is_not_an_ordinary_call():
    call = _native.torch_call()
    assert call, "the extension is built together with the library"
    a, b = torch.zeros(4, 3), torch.zeros(5, 3)
    assert call.cdist(a, b, None, 2.0, False) is None                       # not on a CUDA device
    assert call.cdist(a.numpy(), b, None, 2.0, False) is None
    assert call.cdist(a, b, None, "2", False) is None
    assert call.run_kernel(object(), a, b, *[None] * 7, 0, 0) is None
    assert call.cdist_grad(a, b, b, a, None, 2.0, None) is None


def test_an_extension_of_another_torch_is_not_used(monkeypatch):
    assert _native.torch_call().torch_version == torch.__version__
    monkeypatch.setattr(_native, "_call", None)
    monkeypatch.setattr(torch, "__version__", "0.0.1")
    with pytest.warns(RuntimeWarning, match="built for torch"):
        assert _native.torch_call() is False


def test_enum_classes_that_do_not_match_the_c_abi_are_refused(monkeypatch):
    from kermac_b200 import build_a_kernel
    swapped = dict(build_a_kernel._POWER_CODE)
    swapped[kermac.PowerType.ABS], swapped[kermac.PowerType.SQUARE] = _native.POW_SQUARE, _native.POW_ABS
    monkeypatch.setattr(build_a_kernel, "_POWER_CODE", swapped)
    with pytest.raises(_native.NativeLibraryError, match="PowerType"):
        _native._bind_torch_call(_native.torch_call(), _native.lib())


def _col(t):
    return t.transpose(-1, -2).contiguous().transpose(-1, -2)


@pytest.mark.gpu
@pytest.mark.parametrize("L", [1, 3])
@pytest.mark.parametrize("layout", ["row", "col"])
def test_same_bits_as_the_ctypes_marshalling(L, layout, capsys):
    g = torch.Generator().manual_seed(5)
    def gen(*shape):
        return torch.randn(*((L,) + shape if L > 1 else shape), generator=g).cuda()
    M, N, K, O = 70, 33, 12, 3
    a, b = gen(M, K), gen(N, K)[:1] if L > 1 else gen(N, K)                  # b broadcasts over the batch
    if layout == "col":
        a, b = _col(a), _col(b)
    c, ga, gb, gc, gd = gen(O, M), gen(K, M).abs(), gen(N, K), gen(O, K), gen(N, M)
    bw = torch.full((L,), 3.0, device="cuda")
    gauss = kermac.KernelDescriptor(kermac.InnerOperator.DIFF, kermac.PowerType.SQUARE, kermac.PowerType.NOOP,
                                    kermac.KernelType.GAUSSIAN)
    out = torch.empty(L, M, N, device="cuda")
    calls = [
        lambda **k: kermac.cdist(a, b, **k), lambda **k: kermac.cdist(a, b, p=1, **k),
        lambda **k: kermac.cdist(a, b, p=1.3, out=_col(out), **k), lambda **k: kermac.cdist(a, b, p=2.0, skip_epilogue=True, **k),
        lambda **k: kermac.run_kernel(kermac.kernel_descriptor_laplace_l1, a, b, bandwidth=bw, **k),
        lambda **k: kermac.run_kernel(gauss, a, b, bandwidth=2.0, epsilon=1e-3, regularization=0.5, regularization_offset_x=4, **k),
        lambda **k: kermac.run_kernel(kermac.kernel_descriptor_p_norm, a, b, inner_p=1.5, outer_p=0.5, **k),
        lambda **k: kermac.run_kernel(kermac.kernel_descriptor_mma, a, b, **k),
        lambda **k: kermac.cdist_grad(ga, gb, gc, gd, p=1.5, **k), lambda **k: kermac.cdist_grad(ga, gb, gc, gd, p=1.0, **k),
        lambda **k: kermac.kernel_matvec(kermac.kernel_descriptor_laplace_l2, a, b, c, bandwidth=bw, **k),
    ]
    for call in calls:
        fast, slow = call(), call(debug=True)
        assert "Kermac Debug" in capsys.readouterr().out
        assert fast.shape == slow.shape and torch.equal(fast, slow)
    assert kermac.cdist(a, b, out=out) is out


@pytest.mark.gpu
def test_a_named_contraction_takes_the_native_path(capsys):
    g = torch.Generator().manual_seed(6)
    a, b, c = (torch.randn(*s, generator=g).cuda() for s in ((500, 9), (70, 9), (3, 500)))
    call, tail = _native.torch_call(), (None,) * 3 + (8.0, None, None, 0, 0, 0)
    desc = kermac.kernel_descriptor_laplace_l2
    seen = {}
    for name in (None, "auto", "tensor", "fp32"):
        seen[name] = call.kernel_matvec(desc, a, b, c, None, *tail, name)
        assert torch.equal(seen[name], kermac.kernel_matvec(desc, a, b, c, bandwidth=8.0, contraction=name, debug=True))
    assert torch.equal(seen["auto"], seen["tensor"]) and not torch.equal(seen["fp32"], seen["tensor"])
    for name in ("fp64", "FP32", 1):                         # other spellings are the Python layer's business
        assert call.kernel_matvec(desc, a, b, c, None, *tail, name) is None
    assert torch.equal(kermac.kernel_matvec(desc, a, b, c, bandwidth=8.0, contraction="FP32"), seen["fp32"])
    for name in ("fp64", 1):
        with pytest.raises(ValueError, match="contraction"):
            kermac.kernel_matvec(desc, a, b, c, bandwidth=8.0, contraction=name)


@pytest.mark.gpu
@pytest.mark.parametrize("p", [1.0, 2.0, 1.3])
def test_both_paths_pack_large_row_operands(p, capsys, monkeypatch):
    a, b = torch.randn(6001, 701, device="cuda"), torch.randn(6001, 701, device="cuda")
    with_scratch = []
    launch = _native.launch_build
    monkeypatch.setattr(_native, "launch_build", lambda args, stream, scratch=None:
                        (with_scratch.append(scratch is not None), launch(args, stream, scratch)))
    fast, slow = kermac.cdist(a, b, p=p), kermac.cdist(a, b, p=p, debug=True)
    assert with_scratch == [True] and torch.equal(fast, slow)
    printed = capsys.readouterr().out
    size = 2 * 6016 * 701 * 4
    assert f"with {size} bytes of scratch: operands packed" in printed and f"scratch bytes={size}" in printed
    for debug in (False, True):                              # a full device does without, for the same bits
        slow.fill_(-1.0)
        with full_device():
            kermac.cdist(a, b, out=slow, p=p, debug=debug)
        assert torch.equal(fast, slow)
    assert with_scratch == [True, False] and "scratch bytes=0" in capsys.readouterr().out


@pytest.mark.gpu
def test_exceptions_of_the_python_layer_still_apply():
    a, b = torch.zeros(4, 3, device="cuda"), torch.zeros(5, 3, device="cuda")
    with pytest.raises(ValueError, match="K dimensions must match"):
        kermac.cdist(a, b[:, :2].contiguous())
    with pytest.raises(TypeError, match="float32"):
        kermac.cdist(a.double(), b)
    with pytest.raises(ValueError, match="non-standard memory layout"):
        kermac.cdist(torch.zeros(4, 6, device="cuda")[:, ::2], b)
    with pytest.raises(ValueError, match="must be on a CUDA device"):
        kermac.cdist(a, b.cpu())
    with pytest.raises(ValueError, match="contraction"):
        kermac.cdist_grad(torch.zeros(3, 4, device="cuda"), b, b[:2], torch.zeros(5, 4, device="cuda"), contraction="no")


SLOW_ENTRY_POINTS = """
#include <unistd.h>
#include <stdint.h>
int kermac_b200_build_kernel_scratch(const void* a, void* s, int64_t n, void* st) { usleep(300000); return 0; }
int64_t kermac_b200_build_scratch_bytes(const void* a) { return 0; }
int kermac_b200_cdist_grad(const void* a, void* st) { usleep(300000); return 0; }
int64_t kermac_b200_cdist_grad_scratch_bytes(const void* a) { return 0; }
int kermac_b200_kernel_matvec(const void* a, void* st) { usleep(300000); return 0; }
int64_t kermac_b200_kernel_matvec_scratch_bytes(const void* a) { return 0; }
"""


@pytest.mark.gpu
def test_other_python_threads_run_while_a_call_is_in_its_native_part(tmp_path):
    # entry points that only sleep stand in for a launch that waits on a full queue
    (tmp_path / "slow.c").write_text(SLOW_ENTRY_POINTS)
    subprocess.run(["gcc", "-shared", "-fPIC", str(tmp_path / "slow.c"), "-o", str(tmp_path / "slow.so")], check=True)
    a, b, c = (torch.zeros(n, 4, device="cuda") for n in (5, 6, 3))
    z, cm = torch.zeros(6, 5, device="cuda"), torch.zeros(2, 5, device="cuda")
    call = _native.torch_call()
    calls = (lambda: call.cdist(a, b, None, 2.0, False),
             lambda: call.run_kernel(kermac.kernel_descriptor_l1_norm, a, b, *[None] * 7, 0, 0),
             lambda: call.cdist_grad(a.t().contiguous(), b, c, z, None, 2.0, 0),
             lambda: call.kernel_matvec(kermac.kernel_descriptor_l1_norm, a, b, cm, *[None] * 7, 0, 0, 0, None))
    ticks, stop = [], threading.Event()

    def tick():
        while not stop.is_set():
            ticks.append(time.perf_counter())
            time.sleep(0.005)

    other = threading.Thread(target=tick)
    _native._bind_torch_call(call, ctypes.CDLL(str(tmp_path / "slow.so")))
    try:
        other.start()
        for one in calls:
            began = time.perf_counter()
            assert one() is not None
            ended = time.perf_counter()
            assert ended - began >= 0.3
            assert sum(began + 0.05 < t < ended - 0.05 for t in ticks) >= 5
    finally:
        stop.set()
        other.join()
        _native._bind_torch_call(call, _native.lib())
