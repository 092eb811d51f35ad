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


@pytest.mark.parametrize("hidden,inter", [(3072, 6144), (2560, 4352)])
def test_one_token_feed_forward_chain_on_shared_buffers(backend, hidden, inter):
    """Norm + quantise, gate_up, SwiGLU + quantise, down at one token; tiles and clusters in the first case, the GEMV, which
    reads its weights ahead of its wait, in the second."""
    gen = torch.Generator(device="cuda").manual_seed(hidden)
    w = [(*weight(backend, gen, 2 * inter, hidden), *weight(backend, gen, hidden, inter)) for _ in range(2)]
    xs, residual, norm = rows(gen, 4, hidden), rows(gen, hidden), rows(gen, hidden) * 0.1
    q = backend.rmsnorm_nvfp4_quantize(xs[0], norm, residual, 1e-6, 0.37, False, True)
    gate_up = torch.zeros((1, 2 * inter), dtype=torch.bfloat16, device="cuda")
    act = backend.swiglu_nvfp4_quantize(gate_up[0, :inter], gate_up[0, inter:], 0.11)
    out = torch.empty((1, hidden), dtype=torch.bfloat16, device="cuda")

    def block(i, settle):
        w1, sf1, w2, sf2 = w[i % 2]
        backend.rmsnorm_nvfp4_quantize(xs[i % 4], norm, residual, 1e-6, 0.37, False, True, q)
        settle()
        backend.nvfp4_gemm(w1, sf1, q[2], q[3], 5e-4, 2 * inter, 1, hidden, gate_up)
        settle()
        backend.swiglu_nvfp4_quantize(gate_up[0, :inter], gate_up[0, inter:], 0.11, *act)
        settle()
        backend.nvfp4_gemm(w2, sf2, act[0], act[1], 5e-4, hidden, 1, inter, out)
        settle()

    want = torch.empty((4, 1, hidden), dtype=torch.bfloat16, device="cuda")
    for i in range(4):
        block(i, torch.cuda.synchronize)
        want[i] = out
    wrong = torch.zeros((), dtype=torch.int64, device="cuda")
    for i in range(40):
        block(i, lambda: None)
        wrong += (out != want[i % 4]).sum()
    assert wrong.item() == 0 and out.float().abs().max().item() > 0.1
    assert backend.lib.qwen36_nvfp4_gemm_last_error() == 0 and backend.lib.qwen36_nvfp4_gemv_mma_last_error() == 0


def test_guard_and_argmax_chain_on_shared_buffers(backend):
    """FP8 logits, top-8 guard, and the bf16 argmax of the rows it did not certify (clear, scan, result), over and over into the
    same logits, tokens and flags; ten rows, so that the argmax scans in two passes, of which some have nothing to do."""
    gen = torch.Generator(device="cuda").manual_seed(3)
    vocab, hidden, n = 20000, 1024, 10
    wb = torch.empty((vocab, hidden), dtype=torch.bfloat16, device="cuda").normal_(0.0, 0.02, generator=gen)
    w8, scales = backend.lm_head_fp8_quantize(wb)
    xs = torch.randn((4, n, hidden), generator=gen, device="cuda")
    pick = torch.randint(0, vocab, (4, n), generator=gen, device="cuda")
    boost = torch.full((4, n, 1), 10.0, device="cuda")
    boost[1] = 0.0                                   # no row certified, rows 2 and 9, all certified, the second pass alone
    boost[2, [2, 9]] = 0.0
    boost[0, 8:] = 0.0
    xs = (xs + boost * wb[pick].float() / (0.02 * hidden ** 0.5)).to(torch.bfloat16)
    logits = torch.empty((n, vocab), dtype=torch.bfloat16, device="cuda")

    def step(i, settle):
        backend.lm_head_fp8_gemv(w8, scales, xs[i % 4], logits)
        settle()
        tokens, flags = backend.lm_head_top8_rescore(logits, wb, xs[i % 4], 2.0)
        settle()
        backend.bf16_matvec_argmax_rows(xs[i % 4], wb, tokens, flags)
        settle()
        return torch.stack((tokens, flags))

    want = torch.stack([step(i, torch.cuda.synchronize) for i in range(4)])
    got = torch.stack([step(i, lambda: None) for i in range(40)])
    torch.cuda.synchronize()
    assert torch.equal(got, want.repeat(10, 1, 1))
    flags = want[:, 1].ne(0)
    assert flags[3].all() and not flags[1].any() and flags[2].sum() == 8 and flags[0, :8].all() and not flags[0, 8:].any()
    full = torch.stack([(x.float() @ wb.float().T).argmax(1) for x in xs])
    assert (want[:, 0] == full).float().mean() > 0.9                   # near ties of unpeaked rows aside
