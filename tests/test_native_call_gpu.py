"""The native call (csrc/torch_call.cpp) takes ordinary eager calls and leaves every other one to the Python path."""
import threading

import pytest
import torch

import hf_kernels_helion_b200 as pkg
from hf_kernels_helion_b200 import deep_gemm, runtime
from oracle import fp8_oracle as oracle

pytestmark = pytest.mark.gpu


@pytest.fixture()
def operands(device):
    A, B, As, Bs = [t.to(device) for t in oracle.make_quantised_inputs(48, 384, 512, 1)]
    pkg.w8a8_block_fp8_matmul(A, B, As, Bs, [128, 128])     # binds the module, makes the status word
    return A, B, As, Bs


def _native(A, B, As, Bs, block=None, dtype=torch.float32):
    return runtime.native.matmul(A, B, As, Bs, [128, 128] if block is None else block, dtype)


def test_takes_the_ordinary_call_and_gives_the_same_bits(device, operands):
    A, B, As, Bs = operands
    for dtype in (torch.float32, torch.bfloat16):
        assert torch.equal(_native(*operands, dtype=dtype), runtime.gemm(A, B, As, Bs, 128, 128, dtype))
        assert torch.equal(_native(*operands, block=(128, 128), dtype=dtype), runtime.gemm(A, B, As, Bs, 128, 128, dtype))
    Bs_row = Bs.repeat_interleave(128, 0).contiguous()
    assert torch.equal(_native(A, B, As, Bs_row, 128, torch.bfloat16), runtime.gemm_rowscale(A, B, As, Bs_row, 128, torch.bfloat16))
    wide = torch.randn(48, 1024, device=device).to(torch.bfloat16)
    for x in (wide[:, :512], wide[:, 512:].contiguous(), wide[:1, :512]):       # a strided view, a packed one, one row
        q, s = runtime.native.act_quant(x, 128)
        rq, rs = runtime.quant_act(x, 128)
        assert torch.equal(q.view(torch.uint8), rq.view(torch.uint8)) and torch.equal(s, rs)
        y = runtime.native.linear(x, B, Bs, torch.bfloat16)
        assert torch.equal(y, runtime.linear(x, B, Bs, torch.bfloat16)) and y.shape == (x.shape[0], 384)
    big = torch.randn(3, 100, 512, device=device).to(torch.bfloat16)            # over 256 rows: two launches, three dimensions
    y = runtime.native.linear(big, B, Bs, torch.float32)
    q, s = runtime.quant_act(big.view(300, 512), 128)
    assert torch.equal(y.view(300, 384), runtime.gemm(q, B, s, Bs, 128, 128, torch.float32))
    q, s = runtime.native.weight_quant(wide[:, 8:520], 128)                     # 16-byte, not 32-byte aligned
    rq, rs = runtime.quant_weight(wide[:, 8:520], 128)
    assert torch.equal(q.view(torch.uint8), rq.view(torch.uint8)) and torch.equal(s, rs)
    runtime.check_device_status()


def test_leaves_other_calls_to_the_python_path(device, operands, monkeypatch):
    A, B, As, Bs = operands
    assert _native(A.cpu(), B, As, Bs) is None                                   # another device
    assert _native(A, B, As.double(), Bs) is None                                # a type, shapes, block sizes, a result type
    assert _native(A, B[:, :256], As, Bs) is None and _native(A, B, As[:, :2], Bs) is None
    assert _native(A, B, As, Bs, block=[128, 64]) is None and _native(A, B, As, Bs, block=64) is None
    assert _native(A, B, As, Bs, block=True) is None and _native(A, B, As, Bs, block=1 << 80) is None
    assert _native(A, B, As, Bs, dtype=torch.float16) is None
    assert _native(A[:0], B, As[:0], Bs) is None                                 # empty
    assert _native(A.t().contiguous().t(), B, As, Bs) is None                    # column-major
    assert _native(A, B, As.requires_grad_(), Bs) is None                        # would be recorded
    with torch.no_grad():
        assert _native(A, B, As, Bs) is not None
    As.requires_grad_(False)

    class Sub(torch.Tensor):
        pass

    assert _native(A, B, As.as_subclass(Sub), Bs) is None                        # a subclass, a mode, a transform
    from torch.utils._python_dispatch import TorchDispatchMode

    class Mode(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            return func(*args, **(kwargs or {}))

    with Mode():
        assert _native(A, B, As, Bs) is None
    with torch.device("cuda"):
        assert _native(A, B, As, Bs) is None
    with torch.autograd.forward_ad.dual_level():
        assert _native(A, B, torch.autograd.forward_ad.make_dual(As, As), Bs) is None
    seen = []
    torch.func.vmap(lambda s: (seen.append(_native(A, B, s, Bs)), s)[1])(As.expand(2, *As.shape))
    assert seen == [None]
    monkeypatch.setenv("B200FP8_VARIANT", "tile256")
    assert _native(A, B, As, Bs) is None
    assert runtime.native.act_quant(torch.zeros(4, 130, device=device, dtype=torch.bfloat16), 128) is None
    with pytest.raises(ValueError):
        pkg.w8a8_block_fp8_matmul(A, B, As, Bs, [128, 64])
    with pytest.raises(RuntimeError):
        deep_gemm.gemm_fp8_fp8_bf16_nt(A.cpu(), B.cpu(), As.cpu(), Bs.repeat_interleave(128, 0).cpu())


def test_threads_and_streams(device):
    """Each call has scratch of its own: products of one thread per stream, over shapes that split K, stay right."""
    cases = []
    for i, (M, N, K) in enumerate([(64, 256, 2048), (512, 512, 2048), (16, 1024, 4096), (300, 384, 1664)]):
        A, B, As, Bs = [t.to(device) for t in oracle.make_quantised_inputs(M, N, K, i)]
        cases.append(((A, B, As, Bs), pkg.w8a8_block_fp8_matmul(A, B, As, Bs, [128, 128])))
    torch.cuda.synchronize()
    wrong = []

    def work(i):
        ops, want = cases[i]
        with torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(50):
                if not torch.equal(pkg.w8a8_block_fp8_matmul(*ops, [128, 128]), want):
                    wrong.append(i)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(cases))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert wrong == []
    runtime.check_device_status()


def test_graph_capture(device, operands):
    A, B, As, Bs = operands
    want = pkg.w8a8_block_fp8_matmul(A, B, As, Bs, [128, 128])
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        out = pkg.w8a8_block_fp8_matmul(A, B, As, Bs, [128, 128])
    out.zero_()
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, want)


HOLD = r"""
#include <time.h>
volatile int entered, released;
/* stands in for a library call that takes its time: at most one second, less if somebody sets `released` meanwhile */
int hold(void) {
  struct timespec ms = {0, 1000000};
  int i;
  entered = 1;
  for (i = 0; i < 1000 && !released; ++i) nanosleep(&ms, 0);
  return released ? 0 : 10;
}
"""


def test_other_threads_run_while_a_call_is_in_the_library(device, operands, tmp_path):
    """A launch can wait (a full queue, an allocation), and what it waits for may need another Python thread: the call gives
    the interpreter up meanwhile, as the registered ops do."""
    import ctypes
    import subprocess
    import time

    from hf_kernels_helion_b200 import _lib

    A, B, As, Bs = operands
    (tmp_path / "hold.c").write_text(HOLD)
    subprocess.run(["gcc", "-shared", "-fPIC", "-O1", "-o", str(tmp_path / "hold.so"), str(tmp_path / "hold.c")], check=True)
    held = ctypes.CDLL(str(tmp_path / "hold.so"))
    entered, released = (ctypes.c_int.in_dll(held, n) for n in ("entered", "released"))
    x = torch.zeros(4, 512, device=device, dtype=torch.bfloat16)
    calls = [lambda: _native(A, B, As, Bs), lambda: _native(A, B, As, Bs.repeat_interleave(128, 0), 128, torch.bfloat16),
             lambda: runtime.native.linear(x, B, Bs, torch.bfloat16), lambda: runtime.native.act_quant(x, 128),
             lambda: runtime.native.weight_quant(x, 128)]
    hold = ctypes.cast(held.hold, ctypes.c_void_p).value
    size = [ctypes.cast(getattr(_lib.load(), f"b200fp8_{n}_workspace_bytes"), ctypes.c_void_p).value
            for n in ("gemm", "gemm_rowscale", "linear")]

    def let_go():
        while not entered.value and time.monotonic() < limit:
            time.sleep(0.001)
        released.value = 1

    results = []
    try:
        runtime.native.bind(hold, size[0], hold, size[1], hold, size[2], hold, hold)
        for call in calls:
            entered.value = released.value = 0
            limit = time.monotonic() + 5
            other = threading.Thread(target=let_go)
            other.start()
            results.append(call() is not None)
            other.join()
    finally:
        _lib.load_native()      # binds the library again
    assert results == [True] * len(calls)
    assert torch.equal(_native(*operands), runtime.gemm(A, B, As, Bs, 128, 128, torch.float32))


def test_calls_work_without_the_module(device, operands, monkeypatch):
    """No module that fits (warned about once): the registered ops, the same bits."""
    from hf_kernels_helion_b200 import _lib

    A, B, As, Bs = operands
    want = _native(*operands)
    x = torch.randn(48, 512, device=device).to(torch.bfloat16)
    q, s = runtime.native.act_quant(x, 128)
    tried = []
    monkeypatch.setattr(runtime, "native", None)
    monkeypatch.setattr(runtime, "_native_missing", False)
    monkeypatch.setattr(_lib, "load_native", lambda: tried.append(1))
    for _ in range(2):
        assert torch.equal(pkg.w8a8_block_fp8_matmul(A, B, As, Bs, [128, 128]), want)
        rq, rs = pkg.fp8_act_quant(x)
        assert torch.equal(q.view(torch.uint8), rq.view(torch.uint8)) and torch.equal(s, rs)
    assert tried == [1] and runtime.native is None
