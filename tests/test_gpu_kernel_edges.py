"""Edges of the kernels that a call's sizes select: tiles that are not full, remainders along K, the smallest and the
largest sizes of a choice.  Bar: the bits of the CPU oracle."""
import numpy as np
import pytest

from helpers import bits, rel_err
from oracle import orc

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx(rmi):
    c = rmi.context(0)
    c.set_semantics(rmi.SEM_AVX2)
    yield c
    c.set_prefill_exact(False)


# one shape at least for every CTA tile of the eight-lane tensor-core matmul (4, 8, 16, 32 activation rows), K of one
# block, of a partial and of several chunks
@pytest.mark.parametrize("m,n,k", [(5, 1, 32), (9, 130, 544), (17, 2555, 96), (31, 2560, 1056), (48, 6144, 64), (32, 6130, 160),
                                   (150, 6159, 416)])
def test_eight_lane_matmul_on_tensor_cores(rmi, ctx, m, n, k):
    wb = rmi.synth.q8_0_weight(n, k, seed=m + k)
    w = rmi.QuantizedTensor.from_bytes(wb, rmi.GGML_Q8_0, k, n)
    x = rmi.synth.normal((m, k), seed=n)
    x[m // 2] = 0.0
    ctx.set_prefill_exact(True)
    got = rmi.matmul_q8_0(w, x)
    ctx.set_prefill_exact(False)
    assert np.array_equal(bits(got), bits(orc.q8_forward_batched(wb, x, k, n, orc.SEM_AVX2, threads=8)))
    w.free()


# quantize and GEMV in one kernel (1, 2 and 4 rows up to its longest K), and the row counts around it
@pytest.mark.parametrize("m,n,k", [(1, 1, 32), (1, 4097, 8192), (2, 100, 4096), (4, 33, 2048), (4, 16, 2080), (3, 48, 96)])
@pytest.mark.parametrize("offset", [0, 1])
def test_few_rows_from_device_pointers(rmi, ctx, m, n, k, offset):
    torch = pytest.importorskip("torch")
    wb = rmi.synth.q8_0_weight(n, k, seed=k)
    w = rmi.QuantizedTensor.from_bytes(wb, rmi.GGML_Q8_0, k, n)
    x = rmi.synth.normal((m, k), seed=m)
    d = torch.zeros(m * k + 4, device="cuda")
    d[offset:offset + m * k] = torch.from_numpy(x.reshape(-1)).cuda()      # on a 16-byte boundary, and off one
    out = torch.empty(m * n, device="cuda")
    torch.cuda.synchronize()
    rmi.matmul_q8_0_dev(w, d.data_ptr() + 4 * offset, m, out.data_ptr())
    ctx.sync()
    assert np.array_equal(bits(out.cpu().numpy().reshape(m, n)), bits(orc.q8_forward_batched(wb, x, k, n, orc.SEM_AVX2)))
    w.free()


# Q4_0 and Q6_K through one trait call: row counts on both sides of the kernels' row tiles, ragged output rows
@pytest.mark.parametrize("kind,m,n,k", [("q4_0", 1, 17, 32), ("q4_0", 7, 130, 96), ("q4_0", 8, 64, 1024), ("q4_0", 25, 33, 2080),
                                        ("q6_k", 1, 1, 256), ("q6_k", 3, 37, 512), ("q6_k", 9, 16, 1024), ("q6_k", 2, 5000, 256)])
def test_kernel_trait_forward_batched(rmi, ctx, kind, m, n, k):
    wb = getattr(rmi.synth, kind + "_weight")(n, k, seed=n + k)
    kern = (rmi.Q4_0Kernel if kind == "q4_0" else rmi.Q6_KKernel).new(wb, k, n)
    x = rmi.synth.normal((m, k), seed=m)
    got = np.full((m, n), np.nan, np.float32)
    kern.forward_batched(x, got, k, n)
    for t in range(m):
        if kind == "q4_0":
            ref = orc.q4_0_forward_prequantized(wb, *orc.quantize_q8_0(x[t], orc.SEM_AVX2), k, n)
        else:
            ref = orc.q6k_forward_prepared(wb, x[t], k, n)
        assert np.array_equal(bits(got[t]), bits(ref)), t


# every head size, one to eight query heads per kv head, prompts that end on and beside the edges of row and position tiles
@pytest.mark.parametrize("head_dim,n_head,n_head_kv,positions", [(32, 8, 1, 16), (64, 4, 2, 64), (128, 4, 4, 65), (128, 2, 1, 131)])
def test_prefill_attention_rows_and_heads(rmi, ctx, tmp_path, head_dim, n_head, n_head_kv, positions):
    from tests.synth_model import tiny_cfg
    cfg = tiny_cfg(head_dim=head_dim, n_head=n_head, n_head_kv=n_head_kv)
    path = str(tmp_path / "m.gguf")
    rmi.synth.write_qwen3_gguf(path, cfg, rmi.synth.qwen3_tensors(cfg, 3))
    model = rmi.Qwen3Model.from_file(path)
    prompts = np.stack([rmi.synth.prompt_tokens(cfg["vocab"], positions + 1, seed=b) for b in range(2)])
    s = rmi.Qwen3Session(model, positions + 8, batch=2)
    got = []
    for mode in (rmi.PREFILL_TOKEN_LOOP, rmi.PREFILL_BATCHED):
        s.set_prefill(mode)
        tok = s.generate(prompts, 4)
        got.append((tok, bits(s.hidden()), bits(s.logits())))
    for loop, batched in zip(*got):
        assert np.array_equal(loop, batched)
    s.free()
    model.free()


# Q4_K on the tensor cores: the fewest rows, both CTA widths, rows and super-blocks that fill no tile, chunk or ring
@pytest.mark.parametrize("m,n,k", [(3, 5, 256), (9, 130, 512), (16, 1030, 1280), (33, 2600, 768), (5, 8200, 256), (200, 777, 2304)])
def test_q4_k_on_tensor_cores(rmi, ctx, m, n, k):
    torch = pytest.importorskip("torch")
    wb = rmi.synth.q4_k_weight(n, k, seed=m + n)
    w = rmi.QuantizedTensor.from_bytes(wb, rmi.GGML_Q4_K, k, n)
    x = rmi.synth.normal((m, k), seed=k)
    x[m // 2, : k // 2] = 0.0
    d, out = torch.from_numpy(x).cuda(), torch.empty((m, n), device="cuda")
    torch.cuda.synchronize()
    rmi.matmul_q4_k_q8k_dev(w, d.data_ptr(), m, out.data_ptr())
    ctx.sync()
    ref = np.stack([orc.q4k_forward_prepared(wb, x[t], k, n) for t in range(m)])
    assert np.array_equal(bits(out.cpu().numpy()), bits(ref))
    rmi.matmul_q4_k_dequant_dev(w, d.data_ptr(), m, out.data_ptr())
    ctx.sync()
    ref = x.astype(np.float64) @ orc.dequantize_q4_k_weight(wb, n, k).astype(np.float64).T
    assert rel_err(out.cpu().numpy(), ref.astype(np.float32)) < 2e-6     # no input is rounded, sums are f32
    w.free()
