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
