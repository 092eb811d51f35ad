"""Kernels that start while the kernel ahead drains, called back to back on one stream: what a call reads is complete, and
what it overwrites is no longer read, whatever was called before it.  Every chain runs once without a synchronisation and
is compared, bit for bit, with the same calls synchronised one by one."""
import pytest
import torch

from speedoza_b200 import synth

pytestmark = pytest.mark.gpu


def weight(backend, gen, n, k):
    packed, sf = synth.nvfp4_weight_device(gen, n, k, "cuda")
    return packed, backend.nvfp4_retile_scales(sf)


def rows(gen, *shape):
    return torch.randn(shape, generator=gen, device="cuda").to(torch.bfloat16)


@pytest.mark.parametrize("m,k", [(64, 5120), (1024, 5120), (34816, 5120)])
@pytest.mark.parametrize("tokens", [0, 5, 100])
def test_weight_quantised_ahead_of_its_gemv(backend, m, k, tokens):
    """A matrix is quantised on the device and multiplied by the one-token kernel, which streams its weights before it
    waits for the kernel ahead: directly behind the quantiser, and with a product of other weights in between (split-K form at
    5 tokens, one CTA per tile at 100)."""
    gen = torch.Generator(device="cuda").manual_seed(m + tokens)
    ws = [rows(gen, m, k) for _ in range(3)]
    x, acts = rows(gen, k), rows(gen, max(tokens, 1), k)
    other, other_sf = weight(backend, gen, 1024, k)
    fp4, sf, ts = backend.nvfp4_quantize_rows(ws[0], 0.01)
    a_fp4, a_sf, _ = backend.nvfp4_quantize_rows(acts, 0.01)
    between = torch.empty((max(tokens, 1), 1024), dtype=torch.bfloat16, device="cuda")

    def chain(i, out, settle):
        backend.nvfp4_quantize_rows(ws[i % 3], 0.01, fp4, sf, ts)
        settle()
        if tokens:
            backend.nvfp4_gemm(other, other_sf, a_fp4, a_sf, 1e-4, 1024, tokens, k, between)
            settle()
        backend.nvfp4_matvec(x, fp4, sf, ts, out)
        settle()

    want = torch.empty((3, m), dtype=torch.bfloat16, device="cuda")
    got = torch.empty((24, m), dtype=torch.bfloat16, device="cuda")
    for i in range(3):
        chain(i, want[i], torch.cuda.synchronize)
    for i in range(24):
        chain(i, got[i], lambda: None)
    torch.cuda.synchronize()
    assert torch.equal(got, want.repeat(8, 1)) and not torch.equal(want[0], want[1])


@pytest.mark.parametrize("tokens", [2, 5, 17, 64, 130, 600])
def test_feed_forward_chain_on_shared_buffers(backend, tokens):
    """Quantise, gate_up, SwiGLU + quantise, down; every block overwrites the codes, scales and sums of the block before."""
    gen = torch.Generator(device="cuda").manual_seed(tokens)
    hidden, inter = 2560, 4352
    w = [(*weight(backend, gen, 2 * inter, hidden), *weight(backend, gen, hidden, inter)) for _ in range(2)]
    xs = rows(gen, 4, tokens, hidden)
    q = backend.nvfp4_quantize_rows(xs[0], 0.37)
    gate_up = torch.empty((tokens, 2 * inter), dtype=torch.bfloat16, device="cuda")
    act = backend.swiglu_nvfp4_quantize_rows(gate_up.zero_()[:, :inter], gate_up[:, inter:], 0.11)
    out = torch.empty((tokens, hidden), dtype=torch.bfloat16, device="cuda")

    def block(i, settle):
        w1, sf1, w2, sf2 = w[i % 2]
        backend.nvfp4_quantize_rows(xs[i % 4], 0.37, *q)
        settle()
        backend.nvfp4_gemm(w1, sf1, q[0], q[1], 5e-4, 2 * inter, tokens, hidden, gate_up)
        settle()
        backend.swiglu_nvfp4_quantize_rows(gate_up[:, :inter], gate_up[:, inter:], 0.11, *act)
        settle()
        backend.nvfp4_gemm(w2, sf2, act[0], act[1], 5e-4, hidden, tokens, inter, out)
        settle()

    want = torch.empty((4, tokens, hidden), dtype=torch.bfloat16, device="cuda")
    for i in range(4):
        block(i, torch.cuda.synchronize)
        want[i] = out
    wrong = torch.zeros((), dtype=torch.int64, device="cuda")
    for i in range(40):
        block(i, lambda: None)
        wrong += (out != want[i % 4]).sum()
    assert wrong.item() == 0 and out.float().abs().max().item() > 0.1
