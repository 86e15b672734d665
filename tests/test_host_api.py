"""Host-side mirror of the reference interface: names, argument meaning, error behaviour.
No GPU is needed: every check below fails before a kernel would be launched."""
import inspect

import pytest
import torch

import hf_kernels_helion_b200 as pkg
from hf_kernels_helion_b200 import runtime, tp
from hf_kernels_helion_b200._ops import _OPS_NAME

FP8 = torch.float8_e4m3fn


def _args(M=4, N=128, K=256):
    return (torch.zeros(M, K).to(FP8), torch.zeros(N, K).to(FP8), torch.ones(M, K // 128), torch.ones(N // 128, K // 128))


def test_public_names_and_signature_match_the_reference():
    # torch-ext/finegrained_fp8_helion/__init__.py:7-8 and :17
    assert "w8a8_block_fp8_matmul" in pkg.__all__
    sig = inspect.signature(pkg.w8a8_block_fp8_matmul)
    assert list(sig.parameters) == ["A", "B", "As", "Bs", "block_size", "output_dtype"]
    assert sig.parameters["output_dtype"].default is torch.float32


def test_op_namespace_and_schema_match_the_reference():
    # build/torch-cuda/_ops.py:21-25 and torch-ext/finegrained_fp8_helion/op.py:8-11
    assert _OPS_NAME == "_finegrained_fp8_helion_cuda_b0d7177"
    op = getattr(torch.ops, _OPS_NAME).w8a8_block_fp8_matmul
    schema = str(op.default._schema)
    assert "Tensor A, Tensor B, Tensor As, Tensor Bs, SymInt block_n, SymInt block_k" in schema or \
           "Tensor A, Tensor B, Tensor As, Tensor Bs, int block_n, int block_k" in schema
    assert schema.rstrip().endswith("-> Tensor")


def test_fake_impl_shapes_and_dtypes():
    A, B, As, Bs = [t.to("meta") for t in _args(5, 256, 384)]
    ns = getattr(torch.ops, _OPS_NAME)
    assert ns.w8a8_block_fp8_matmul(A, B, As, Bs, 128, 128).shape == (5, 256)
    assert ns.w8a8_block_fp8_matmul(A, B, As, Bs, 128, 128).dtype == torch.float32   # op.py:16 of the reference
    assert ns.w8a8_block_fp8_matmul_out(A, B, As, Bs, 128, 128, 0).dtype == torch.bfloat16
    q, s = ns.fp8_act_quant(torch.empty(5, 384, dtype=torch.bfloat16, device="meta"), 128)
    assert q.shape == (5, 384) and q.dtype == FP8 and s.shape == (5, 3) and s.dtype == torch.float32


def test_argument_validation():
    A, B, As, Bs = _args()
    with pytest.raises(ValueError, match="block_size"):
        runtime.gemm(A, B, As, Bs, 64, 128, torch.bfloat16)
    with pytest.raises(ValueError, match="output dtype"):
        runtime.gemm(A, B, As, Bs, 128, 128, torch.float16)
    with pytest.raises(ValueError, match="float8_e4m3fn"):
        runtime.gemm(A.float(), B, As, Bs, 128, 128, torch.bfloat16)
    with pytest.raises(ValueError, match="float32"):
        runtime.gemm(A, B, As.double(), Bs, 128, 128, torch.bfloat16)
    with pytest.raises(ValueError, match="As must be"):
        runtime.gemm(A, B, As[:, :1], Bs, 128, 128, torch.bfloat16)
    with pytest.raises(ValueError, match="Bs must be"):
        runtime.gemm(A, B, As, torch.ones(128, 2), 128, 128, torch.bfloat16)   # legacy per-row scales are rejected
    with pytest.raises(ValueError, match="K="):
        runtime.gemm(A, B[:, :128], As, Bs, 128, 128, torch.bfloat16)
    with pytest.raises(ValueError, match="2-D"):
        runtime.gemm(A[0], B, As, Bs, 128, 128, torch.bfloat16)
    with pytest.raises(ValueError, match="unknown variant"):
        runtime.resolve_variant("fastest")


def test_no_cpu_fallback():
    A, B, As, Bs = _args()
    with pytest.raises(RuntimeError, match="no CPU implementation"):
        pkg.w8a8_block_fp8_matmul(A, B, As, Bs, [128, 128], torch.bfloat16)
    with pytest.raises(RuntimeError, match="no CPU implementation"):
        pkg.fp8_act_quant(torch.zeros(4, 128, dtype=torch.bfloat16))
    with pytest.raises(ValueError, match="bfloat16"):
        pkg.fp8_act_quant(torch.zeros(4, 128))
    with pytest.raises(ValueError, match="multiple of 8"):
        pkg.fp8_act_quant(torch.zeros(4, 100, dtype=torch.bfloat16))


def test_missing_library_fails_loudly(monkeypatch, tmp_path):
    from hf_kernels_helion_b200 import _lib

    monkeypatch.setattr(_lib, "_lib", None)
    monkeypatch.setattr(_lib, "LIB_PATH", tmp_path / "libb200fp8.so")
    with pytest.raises(RuntimeError, match="no non-CUDA fallback"):
        _lib.load()


def test_product_code_never_imports_the_oracle():
    import pathlib

    root = pathlib.Path(pkg.__file__).parent
    for f in list(root.rglob("*.py")) + list(root.rglob("*.cu")) + list(root.rglob("*.cuh")):
        assert "oracle" not in f.read_text(), f"{f} mentions the oracle"


def test_shard_bounds():
    assert tp.shard_bounds(18432, 8, 3) == (6912, 9216)
    assert tp.shard_bounds(18432, 1, 0) == (0, 18432)
    with pytest.raises(ValueError):
        tp.shard_bounds(18432 + 128, 8, 0)
    B = torch.arange(512 * 4).reshape(512, 4)
    Bs = torch.arange(4 * 1).reshape(4, 1)
    b, bs = tp.shard_weight(B, Bs, 2, 1)
    assert torch.equal(b, B[256:]) and torch.equal(bs, Bs[2:])


def test_native_module_is_optional(lib, monkeypatch):
    """Without a native call module that this torch and this Python can use, the calls keep the way through the registered ops;
    one that was built for others is never called."""
    import sys
    import types

    from hf_kernels_helion_b200 import _lib

    name = "hf_kernels_helion_b200._torch_call"
    monkeypatch.delattr(pkg, "_torch_call", raising=False)
    monkeypatch.setitem(sys.modules, name, None)                     # no file, or one that does not load
    with pytest.warns(RuntimeWarning, match="does not load"):
        assert _lib.load_native() is None

    def never(*args):
        raise AssertionError("called")

    for other in (types.SimpleNamespace(bind=never, built_for="torch 1.0, Python 2.7"), types.SimpleNamespace(bind=never)):
        monkeypatch.setitem(sys.modules, name, other)
        monkeypatch.setattr(pkg, "_torch_call", other, raising=False)
        with pytest.warns(RuntimeWarning, match="was built for"):
            assert _lib.load_native() is None


def test_native_module_is_rebuilt_for_another_torch(lib, monkeypatch):
    from hf_kernels_helion_b200 import _lib, build

    assert not build.is_stale()
    monkeypatch.setattr(_lib, "native_tag", lambda: "torch 1.0, Python 2.7")
    assert build.is_stale()


def test_fake_cuda_tensors_need_no_library(monkeypatch, tmp_path):
    """Tracing with fake CUDA tensors gives shapes and types where the library has not been built."""
    from torch._subclasses.fake_tensor import FakeTensorMode

    from hf_kernels_helion_b200 import _lib, deep_gemm

    monkeypatch.setattr(_lib, "_lib", None)
    monkeypatch.setattr(_lib, "LIB_PATH", tmp_path / "libb200fp8.so")
    monkeypatch.setattr(runtime, "native", None)
    monkeypatch.setattr(runtime, "_native_missing", False)
    with FakeTensorMode():
        A, B, As, Bs = [t.to("cuda") for t in _args(5, 256, 384)]
        out = pkg.w8a8_block_fp8_matmul(A, B, As, Bs, [128, 128], torch.bfloat16)
        assert out.shape == (5, 256) and out.dtype == torch.bfloat16 and out.is_cuda
        q, s = pkg.fp8_act_quant(torch.empty(5, 384, dtype=torch.bfloat16, device="cuda"))
        assert q.shape == (5, 384) and q.dtype == FP8 and s.shape == (5, 3)
        out = deep_gemm.gemm_fp8_fp8_bf16_nt(A, B, As, Bs.repeat_interleave(128, 0))
        assert out.shape == (5, 256) and out.dtype == torch.bfloat16
    assert runtime.native is None and not runtime._native_missing


def test_two_first_calls_agree_on_the_status_word(monkeypatch):
    """Two threads' first calls on a device: one word for both and for the native call module. A word that only one of them
    knew would be freed while the module still pointed kernels at it."""
    import types

    told, words, theirs = {}, {}, torch.zeros(1, dtype=torch.int32)

    def zeros(*args, **kwargs):      # the other thread is done first while this one allocates
        words[5] = theirs
        return torch.ones(1, dtype=torch.int32)

    monkeypatch.setattr(runtime, "_status_words", words)
    monkeypatch.setattr(runtime, "native", types.SimpleNamespace(set_status=told.__setitem__))
    monkeypatch.setattr(runtime, "torch", types.SimpleNamespace(zeros=zeros, int32=torch.int32, device=torch.device))
    assert runtime.status_word(torch.device("cuda", 5)) is theirs and words == {5: theirs}
    assert told == {5: theirs.data_ptr()}


def test_native_module_learns_of_every_status_word(monkeypatch):
    """A word that another thread makes while the module is being set up."""
    import types

    told, theirs = {}, torch.zeros(1, dtype=torch.int32)

    class Words(dict):
        def items(self):             # the other thread makes its word once these have been listed
            listed = list(super().items())
            self[7] = theirs
            if runtime.native is not None:
                runtime.native.set_status(7, theirs.data_ptr())
            return listed

    module = types.SimpleNamespace(set_status=told.__setitem__)
    monkeypatch.setattr(runtime, "_status_words", Words())
    monkeypatch.setattr(runtime, "native", None)
    monkeypatch.setattr(runtime, "_native_missing", False)
    monkeypatch.setattr(runtime._lib, "load_native", lambda: module)
    monkeypatch.setattr(runtime._lib, "is_built", lambda: True)
    monkeypatch.setattr(torch.Tensor, "is_cuda", True)
    assert runtime.native_for(torch.zeros(1)) is module
    assert told == {7: theirs.data_ptr()}


def test_kernels_that_start_early_load_what_others_write_with_ordinary_loads():
    """A kernel launched with programmatic serialisation begins before the one in front of it has ended, so its operands are
    not read-only for its lifetime: no __ldg, no ld.global.nc and no const __restrict__ pointer (which the compiler may turn
    into one) where a file's kernels wait for their predecessor."""
    import pathlib
    import re

    waiting = 0
    for f in sorted((pathlib.Path(pkg.__file__).parent / "csrc").glob("*.cuh")):
        text = re.sub(r"//[^\n]*", "", f.read_text())
        if "griddepcontrol.wait" not in text and "pdl_wait" not in text:
            continue
        waiting += 1
        assert "__ldg" not in text and "global.nc" not in text, f.name
        for body in text.split("__global__")[1:]:
            if "griddepcontrol.wait" in body or "pdl_wait" in body:
                assert not re.search(r"const\s+\w+\s*\*\s*__restrict__", body.split("{")[0]), f.name
    assert waiting >= 2
