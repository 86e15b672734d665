"""Launches overlap the end of the kernel before them (programmatic serialisation): nothing may be read or overwritten early."""
import pytest
import torch

import hf_kernels_helion_b200 as pkg
from hf_kernels_helion_b200 import deep_gemm, runtime
from oracle import fp8_oracle as oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K", [(4, 2560, 2048), (64, 512, 512), (300, 384, 1664), (512, 512, 2048)])
def test_operands_written_by_the_kernel_before(device, M, N, K):
    """Activations, weights and scales produced by the launch right before the call, scratch and results reused call after
    call: the values of a synchronised run, twenty times over with alternating inputs."""
    g = torch.Generator().manual_seed(M + N)
    xs = [torch.randn(M, K, generator=g).to(torch.bfloat16).to(device) for _ in range(2)]
    ws = [(torch.randn(N, K, generator=g) * 0.02).to(torch.bfloat16).to(device) for _ in range(2)]

    def chain(x, w, sync):
        s = torch.cuda.synchronize if sync else (lambda: None)
        q, qs = pkg.fp8_act_quant(x)
        s()
        b, bs = pkg.fp8_weight_quant(w)
        s()
        y = pkg.w8a8_block_fp8_matmul(q, b, qs, bs, [128, 128], torch.bfloat16)
        s()
        z = pkg.fp8_linear(x, b, bs)
        s()
        rb, rs = pkg.fp8_act_quant(w)
        s()
        r = deep_gemm.gemm_fp8_fp8_bf16_nt(q, rb, qs, rs)
        s()
        q2, s2 = pkg.fp8_act_quant(y[:, :N // 128 * 128])       # reads what the matmul wrote
        s()
        return y, z, r, q2.view(torch.uint8), s2

    want = [chain(x, w, True) for x, w in zip(xs, ws)]
    got = [chain(xs[i % 2], ws[i % 2], False) for i in range(20)]
    torch.cuda.synchronize()
    for i, res in enumerate(got):
        for a, b in zip(res, want[i % 2]):
            assert torch.equal(a, b)
    qa, sa = oracle.quant_act(xs[0].cpu())
    qb, sb = oracle.quant_weight(ws[0].cpu())
    assert oracle.bf16_ulp_error(want[0][0].cpu(), oracle.gemm_dequant(qa, qb, sa, sb)) <= 1
    runtime.check_device_status()


def _inputs(device, M, N, K, seed):
    g = torch.Generator().manual_seed(seed)
    return (torch.randn(M, K, generator=g).to(torch.bfloat16).to(device),
            (torch.randn(N, K, generator=g) * 0.02).to(torch.bfloat16).to(device))


def _forward(x, w):
    q, qs = pkg.fp8_act_quant(x)
    b, bs = pkg.fp8_weight_quant(w)
    y = pkg.w8a8_block_fp8_matmul(q, b, qs, bs, [128, 128], torch.bfloat16)
    z = pkg.fp8_linear(x, b, bs)
    rb, rs = pkg.fp8_act_quant(w)
    return y, z, deep_gemm.gemm_fp8_fp8_bf16_nt(q, rb, qs, rs)


@pytest.mark.parametrize("M,N,K", [(4, 2560, 2048), (300, 384, 1664), (1300, 3584, 2064)])
def test_captured_chain(device, M, N, K):
    """The same chain recorded into a graph, replayed over changing inputs without waiting in between."""
    sets = [_inputs(device, M, N, K, s) for s in (1, 2)]
    want = [_forward(x, w) for x, w in sets]
    torch.cuda.synchronize()
    x, w = [t.clone() for t in sets[0]]
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        _forward(x, w)
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = _forward(x, w)
    got = []
    for i in range(10):
        x.copy_(sets[i % 2][0])
        w.copy_(sets[i % 2][1])
        graph.replay()
        got.append([t.clone() for t in out])
    torch.cuda.synchronize()
    for i, res in enumerate(got):
        for a, b in zip(res, want[i % 2]):
            assert torch.equal(a, b)
    runtime.check_device_status()


def test_inputs_made_on_another_stream(device):
    """A call behind an event of another stream starts after what that stream wrote, and the other stream behind an event of
    this one after what the call read."""
    M, N, K = 300, 384, 1664
    sets = [_inputs(device, M, N, K, s) for s in (3, 4)]
    want = [_forward(x, w) for x, w in sets]
    x, w = [t.clone() for t in sets[0]]
    slow = torch.randn(4096, 4096, device=device)
    other = torch.cuda.Stream()
    here = torch.cuda.current_stream()
    torch.cuda.synchronize()
    got = []
    for i in range(8):
        other.wait_stream(here)
        with torch.cuda.stream(other):
            torch.mm(slow, slow)                 # about 2 ms before the operands are there
            x.copy_(sets[i % 2][0])
            w.copy_(sets[i % 2][1])
        here.wait_stream(other)
        got.append(_forward(x, w))
    torch.cuda.synchronize()
    for i, res in enumerate(got):
        for a, b in zip(res, want[i % 2]):
            assert torch.equal(a, b)
    runtime.check_device_status()


def test_one_workspace_for_every_form(device):
    """Calls of the C ABI that share one workspace on one stream, form after form: clusters, split tails on pairs, copied and
    direct scales, fused quantisation, row scales, stream-K."""
    from hf_kernels_helion_b200 import _lib

    lib = _lib.load()
    word, stream = runtime.status_word(device).data_ptr(), torch.cuda.current_stream(device).cuda_stream
    calls, size = [], 0
    for M, N, K, variant in [(512, 512, 2048, 0), (1611, 7008, 4208, 0), (300, 2560, 4096, 7), (64, 2560, 2048, 3),
                             (5, 1280, 1664, 0), (1000, 1304, 1152, 4), (4, 2560, 2048, "linear"), (300, 512, 1664, "row"),
                             (1300, 3584, 2064, "row"), (200, 512, 640, "linear")]:
        x, w = _inputs(device, M, N, K, M + N)
        A, As = pkg.fp8_act_quant(x)
        B, Bs = pkg.fp8_weight_quant(w)
        kb, out = As.shape[1], torch.empty(M, N, device=device)
        if variant == "row":
            B, Bs = pkg.fp8_act_quant(w)
            want = runtime.gemm_rowscale(A, B, As, Bs, 128, torch.float32)
            need = lib.b200fp8_gemm_rowscale_workspace_bytes(M, N, K)
            args = (A.data_ptr(), B.data_ptr(), As.data_ptr(), Bs.data_ptr(), out.data_ptr(), M, N, K, K, K, kb, kb, N, 1)
            call = lib.b200fp8_gemm_rowscale
        elif variant == "linear":
            want = runtime.linear(x, B, Bs, torch.float32)
            need = lib.b200fp8_linear_workspace_bytes(M, N, K, 0)
            args = (x.data_ptr(), B.data_ptr(), Bs.data_ptr(), out.data_ptr(), M, N, K, K, K, kb, N, 1, 0)
            call = lib.b200fp8_linear
        else:
            want = runtime.gemm(A, B, As, Bs, 128, 128, torch.float32, variant=variant)
            need = lib.b200fp8_gemm_workspace_bytes(M, N, K, variant)
            args = (A.data_ptr(), B.data_ptr(), As.data_ptr(), Bs.data_ptr(), out.data_ptr(), M, N, K, K, K, kb, kb, N, 1, variant)
            call = lib.b200fp8_gemm
        assert need >= 0
        size = max(size, need)
        calls.append((call, args, out, want, (x, A, B, As, Bs)))
    ws = torch.empty(size, dtype=torch.uint8, device=device)
    torch.cuda.synchronize()
    for order in (range(len(calls)), reversed(range(len(calls))), [i * 3 % len(calls) for i in range(len(calls))]):
        order = list(order)
        for _ in range(5):
            for i in order:
                call, args, out, _, _ = calls[i]
                out.fill_(7.0)
                assert call(*args, ws.data_ptr(), size, word, stream) == 0
        for call, args, out, _, _ in calls:       # and once without torch's launches in between
            assert call(*args, ws.data_ptr(), size, word, stream) == 0
        torch.cuda.synchronize()
        for _, _, out, want, _ in calls:
            assert torch.equal(out, want)
    runtime.check_device_status()
