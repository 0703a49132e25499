"""Numerics of every CUDA kernel against a plain PyTorch fp32 restatement of the same op.

Metric and thresholds follow the reference's op tests (NMSE; MUL_MAT / FLASH_ATTN_EXT 5e-4:
llama.cpp/tests/test-backend-ops.cpp:273-287,3716-3718,6049-6051)."""
import ctypes
import math

import pytest
import torch

from distributed_llm_pipeline_b200.gguf import GGMLType
from distributed_llm_pipeline_b200.models.reference import apply_rope, nmse
from distributed_llm_pipeline_b200.ops import api as ops
from distributed_llm_pipeline_b200.ops.weights import DeviceWeight

pytestmark = pytest.mark.gpu
DEV = "cuda"
WTYPES = [GGMLType.F16, GGMLType.BF16, GGMLType.Q8_0, GGMLType.Q4_K, GGMLType.Q5_K, GGMLType.Q6_K]


def _w(N, K, t, seed=0):
    g = torch.Generator().manual_seed(seed)
    dense = torch.randn(N, K, generator=g) * 0.05
    w = DeviceWeight.from_dense(dense, t, DEV)
    from distributed_llm_pipeline_b200.gguf.quants import dequantize, quantize
    import numpy as np
    exact = torch.from_numpy(dequantize(quantize(dense.numpy(), t), t, (N, K)).astype(np.float32)).to(DEV)
    return w, exact


@pytest.mark.parametrize("t", WTYPES)
def test_dequant_rows_exact(t):
    w, exact = _w(64, 512, t)
    out = ops.dequant_rows(w, None)
    assert torch.equal(out, exact) or nmse(exact, out) < 1e-9
    rows = torch.tensor([5, 0, 63, 5], dtype=torch.int32, device=DEV)
    assert nmse(exact[rows.long()], ops.dequant_rows(w, rows)) < 1e-9


@pytest.mark.parametrize("t", WTYPES)
@pytest.mark.parametrize("T", [1, 2, 4])
def test_gemv_store_and_add(t, T):
    N, K = 384, 1024
    w, exact = _w(N, K, t, 1)
    x = (torch.randn(T, K, device=DEV) * 2).half()
    ref = x.float() @ exact.T
    y16 = ops.linear(w, x, "f16")
    y32 = ops.linear(w, x, "f32")
    # block-quantised weights use int8 activations + dp4a on the decode path (the reference's q8_1 numerics class;
    # its own MUL_MAT tolerance is 5e-4): allow 5e-5 there, 5e-6 for the dense types
    tol = 5e-5 if t.name.startswith("Q") else 5e-6
    assert nmse(ref, y32) < tol and nmse(ref, y16) < tol
    acc = torch.ones(T, N, device=DEV)
    ops.linear(w, x, "add", out=acc)
    assert nmse(ref + 1, acc) < tol


@pytest.mark.parametrize("t", [GGMLType.F16, GGMLType.Q8_0, GGMLType.Q4_K, GGMLType.Q6_K])
def test_gemv_fused_norm_and_swiglu(t):
    N, K, T = 512, 768, 2
    wg, eg = _w(N, K, t, 2)
    wu, eu = _w(N, K, t, 3)
    h = torch.randn(T, K, device=DEV) * 3
    nw = torch.rand(K, device=DEV) + 0.5
    eps = 1e-5
    xn = (h * torch.rsqrt(h.pow(2).mean(-1, keepdim=True) + eps) * nw).half().float()
    ref = torch.nn.functional.silu(xn @ eg.T) * (xn @ eu.T)
    y = ops.linear(wg, h, "swiglu", w_up=wu, norm_w=nw, eps=eps)
    assert nmse(ref, y) < (2e-4 if t.name.startswith("Q") else 2e-5)


@pytest.mark.parametrize("t", [GGMLType.Q8_0, GGMLType.Q4_K, GGMLType.Q5_K, GGMLType.Q6_K])
@pytest.mark.parametrize("T", [1, 2, 4])
@pytest.mark.parametrize("N,K", [(2, 256), (298, 768), (1002, 2048), (3000, 5632), (640, 14336)])
def test_gemv_quant_of_every_width(t, T, N, K):
    """Fewer rows than blocks, one and several stages of the Q6_K ring of which the last is partial, columns that end inside a warp's round, widths at
    which a stage holds 8 rows down to 1 - plain, with the residual add, and with norm and gate.  The activations are rounded to 8 bits (relative
    to the largest of 32: squared error 2.5e-5 of randn values; the few sums of the smallest shapes scatter by a factor of 10 around it)."""
    (w, exact), (u, exact_u) = _w(N, K, t, 1), _w(N, K, t, 2)
    g = torch.Generator(DEV).manual_seed(N)
    h, norm = torch.randn(T, K, device=DEV, generator=g), torch.rand(K, device=DEV, generator=g) + 0.5
    x = (h * torch.rsqrt(h.pow(2).mean(-1, keepdim=True) + 1e-5) * norm).half()
    ref, up = x.double() @ exact.double().T, x.double() @ exact_u.double().T
    tol = 5e-5 if N * T > 500 else 5e-4
    assert nmse(ref, ops.linear(w, x, "f32")) < tol
    assert nmse(ref + 1, ops.linear(w, x, "add", out=torch.ones(T, N, device=DEV))) < tol
    assert nmse(ref, ops.linear(w, h, "f32", norm_w=norm, eps=1e-5)) < tol
    assert nmse(torch.nn.functional.silu(ref) * up, ops.linear(w, h, "swiglu", w_up=u, norm_w=norm, eps=1e-5)) < 4 * tol


@pytest.mark.parametrize("t", [GGMLType.F16, GGMLType.BF16])
@pytest.mark.parametrize("T", [1, 2, 4])
@pytest.mark.parametrize("N,K", [(6144, 1024), (4736, 2048), (3072, 3584)])
def test_gemv_large_shapes(t, T, N, K):
    """Decode-sized matrices (thousands of rows, the shapes the balanced row ranges / dynamic unit queue are tuned for): every
    epilogue, repeated launches, bit-identical results run to run."""
    w, exact = _w(N, K, t, 5)
    wu, eu = _w(N, K, t, 6)
    x = (torch.randn(T, K, device=DEV) * 2).half()
    ref = x.float() @ exact.T
    for _ in range(3):
        assert nmse(ref, ops.linear(w, x, "f32")) < 5e-6
        assert nmse(ref, ops.linear(w, x, "f16")) < 5e-6
    acc = torch.ones(T, N, device=DEV)
    ops.linear(w, x, "add", out=acc)
    ops.linear(w, x, "add", out=acc)
    assert nmse(2 * ref + 1, acc) < 5e-6
    h = torch.randn(T, K, device=DEV) * 3
    nw = torch.rand(K, device=DEV) + 0.5
    xn = (h * torch.rsqrt(h.pow(2).mean(-1, keepdim=True) + 1e-5) * nw).half().float()
    refs = torch.nn.functional.silu(xn @ exact.T) * (xn @ eu.T)
    for _ in range(2):
        assert nmse(refs, ops.linear(w, h, "swiglu", w_up=wu, norm_w=nw, eps=1e-5)) < 2e-5
    a, b = ops.linear(w, x, "f32"), ops.linear(w, x, "f32")
    assert torch.equal(a, b)            # chunk partials are summed in a fixed order: bit-identical run to run


@pytest.mark.parametrize("T,N,K", [(5, 128, 64), (16, 256, 256), (37, 384, 1024), (128, 512, 512), (300, 128, 2048), (512, 1024, 4096)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_gemm_tcgen05_store(T, N, K, dtype):
    w = (torch.randn(N, K, device=DEV) * 0.05).to(dtype)
    x = torch.randn(T, K, device=DEV).to(dtype)
    ref = x.float() @ w.float().T
    y = torch.empty(T, N, device=DEV, dtype=torch.float32)
    ops.gemm_f16(w, x, y, epilogue=1)
    assert nmse(ref, y) < 1e-6
    y16 = torch.empty(T, N, device=DEV, dtype=torch.float16)
    ops.gemm_f16(w, x, y16, epilogue=0)
    assert nmse(ref, y16) < 5e-6


def test_gemm_tcgen05_ragged_n_splitk_swiglu():
    T, N, K = 70, 200, 1536   # N not a multiple of 128: OOB rows are zero-filled and masked
    w = (torch.randn(N, K, device=DEV) * 0.05).half()
    u = (torch.randn(N, K, device=DEV) * 0.05).half()
    x = torch.randn(T, K, device=DEV).half()
    ref = x.float() @ w.float().T
    acc = torch.full((T, N), 2.0, device=DEV)
    ops.gemm_f16(w, x, acc, epilogue=2, split_k=4)
    assert nmse(ref + 2, acc) < 1e-6
    sw = torch.empty(T, N, device=DEV, dtype=torch.float16)
    ops.gemm_f16(w, x, sw, epilogue=3, w_up=u)
    assert nmse(torch.nn.functional.silu(ref) * (x.float() @ u.float().T), sw) < 5e-6


@pytest.mark.parametrize("T,N,K", [(65, 256, 64), (100, 130, 200), (128, 300, 1024), (257, 512, 2056), (700, 4096, 512), (1030, 2304, 320)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_gemm_on_pairs_of_sms(T, N, K, dtype):
    """The smallest and widest token tiles, row tiles that end inside a pair or inside its second block, columns that are no multiple of 64, one and
    several waves, with every kind of epilogue.  Sums are fp32 (relative 2^-24 sqrt(K)); 16-bit outputs round once more."""
    g = torch.Generator(DEV).manual_seed(7)
    x, w, u = ((torch.randn(n, K, device=DEV, generator=g) * s).to(dtype) for n, s in ((T, 1.0), (N, K ** -0.5), (N, K ** -0.5)))
    ref, up = (x.double() @ m.double().T for m in (w, u))
    y, acc = torch.zeros(T, N, device=DEV), torch.ones(T, N, device=DEV)
    assert nmse(ref, ops.gemm_f16(w, x, y, epilogue=1)) < 1e-11
    assert nmse(ref + 1, ops.gemm_f16(w, x, acc, epilogue=2)) < 1e-11
    assert nmse(ref, ops.gemm_f16(w, x, torch.zeros(T, N, device=DEV, dtype=torch.float16), epilogue=0)) < 1e-7
    assert nmse(torch.nn.functional.silu(ref) * up, ops.gemm_f16(w, x, torch.zeros(T, N, device=DEV, dtype=torch.float16), epilogue=3, w_up=u)) < 2e-7
    if dtype == torch.bfloat16:
        for epi, want in ((4, ref), (6, torch.nn.functional.gelu(ref, approximate="tanh") * up), (7, torch.relu(ref) ** 2), (8, torch.nn.functional.silu(ref) * up)):
            out = ops.gemm_f16(w, x, torch.zeros(T, N, device=DEV, dtype=torch.bfloat16), epilogue=epi, w_up=u if epi in (6, 8) else None)
            assert nmse(want, out) < 6e-6, epi


@pytest.mark.parametrize("t", [GGMLType.Q8_0, GGMLType.Q4_K, GGMLType.Q5_K, GGMLType.Q6_K])
@pytest.mark.parametrize("T,N,K", [(48, 256, 512), (300, 200, 1024), (7, 384, 2048)])
def test_linear_quant_dequant_fused_gemm(t, T, N, K):
    """Block-quant decode fused into the tcgen05 GEMM's A-operand producer (no scratch), all epilogues."""
    w, exact = _w(N, K, t, 4)
    u, exact_u = _w(N, K, t, 5)
    x = torch.randn(T, K, device=DEV).half()
    ref = x.float() @ exact.T
    assert nmse(ref, ops.linear(w, x, "f32")) < 5e-6            # weights are rounded to fp16 after decode
    assert nmse(ref, ops.linear(w, x, "f16")) < 5e-6
    acc = torch.ones(T, N, device=DEV)
    ops.linear(w, x, "add", out=acc)
    assert nmse(ref + 1, acc) < 5e-6
    sw = ops.linear(w, x, "swiglu", w_up=u)
    assert nmse(torch.nn.functional.silu(ref) * (x.float() @ exact_u.T), sw) < 2e-5


@pytest.mark.parametrize("t", [GGMLType.Q8_0, GGMLType.Q4_K, GGMLType.Q5_K, GGMLType.Q6_K])
@pytest.mark.parametrize("T,N,K", [(5, 128, 256), (16, 200, 512), (17, 126, 768), (33, 384, 2304), (64, 130, 4096), (65, 256, 512), (192, 384, 512)])
def test_linear_quant_few_tokens(t, T, N, K):
    """Token tiles of 16, 32 and 64 (and the first size behind them), partial row tiles, one unit of columns up to several splits of K.  The weights
    enter as fp16 values (relative 2^-12 on average, squared 2e-8 with the margin of the few that round the other way); sums are fp32."""
    w, exact = _w(N, K, t, 1)
    u, exact_u = _w(N, K, t, 2)
    x = torch.randn(T, K, device=DEV, generator=torch.Generator(DEV).manual_seed(3)).half()
    ref = x.double() @ exact.double().T
    assert nmse(ref, ops.linear(w, x, "f32")) < 2e-7
    acc = torch.ones(T, N, device=DEV)
    assert nmse(ref + 1, ops.linear(w, x, "add", out=acc)) < 2e-7
    assert nmse(ref, ops.linear(w, x, "f16")) < 4e-7          # (and the rounding of the output)
    assert nmse(torch.nn.functional.silu(ref) * (x.double() @ exact_u.double().T), ops.linear(w, x, "swiglu", w_up=u)) < 2e-6


@pytest.mark.parametrize("T,N,K,t", [(553, 4096, 4096, GGMLType.F16), (1041, 2048, 5632, GGMLType.F16), (1041, 4096, 4096, GGMLType.Q8_0), (7, 9600, 1536, GGMLType.Q4_K),
                                     (40, 2048, 512, GGMLType.Q8_0), (150, 9600, 768, GGMLType.Q6_K)])
def test_residual_sums_repeat(T, N, K, t):
    """Sizes at which the tiles fill the machine: the residual add gives the same bits every time (no atomics of several splits of K), also through the
    workspace, and is right."""
    w = DeviceWeight.from_dense(torch.randn(N, K, generator=torch.Generator().manual_seed(1)) * 0.05, t, DEV)
    x = torch.randn(T, K, device=DEV, generator=torch.Generator(DEV).manual_seed(T)).half()
    base = torch.randn(T, N, device=DEV, generator=torch.Generator(DEV).manual_seed(N))
    runs = [ops.linear(w, x, "add", out=base.clone()) for _ in range(10)]
    assert all(torch.equal(runs[0], r) for r in runs)
    dense = ops.dequant_rows(w, None, out=torch.empty(N, K, device=DEV)) if t.name.startswith("Q") else w.planes[0].view(N, K)
    assert nmse(base.double() + x.double() @ dense.double().T, runs[0]) < 2e-7


def _blocks(t, N, K, seed):
    """Random 4- and 5-bit blocks whose scales and mins lie up to 2^12 apart either way, with zeros and negative ones among them; bytes and 64-bit values."""
    import numpy as np
    g = np.random.default_rng(seed)
    size, n = (144, 8) if t == GGMLType.Q4_K else (176, 8)
    raw = g.integers(0, 256, (N, K // 256, size), dtype=np.uint8)
    d, m = (np.float16(g.uniform(0.5, 2, (N, K // 256)) * 2.0 ** g.integers(-13, -1, (N, K // 256)) * g.choice([1, 1, 1, -1, 0], (N, K // 256))) for _ in range(2))
    raw[..., 0:2], raw[..., 2:4] = d[..., None].view(np.uint8), m[..., None].view(np.uint8)
    s = raw[..., 4:16].astype(np.int64)
    scale = np.concatenate([s[..., :4] & 63, (s[..., 8:] & 15) | (s[..., :4] >> 6 << 4)], -1)
    least = np.concatenate([s[..., 4:8] & 63, (s[..., 8:] >> 4) | (s[..., 4:8] >> 6 << 4)], -1)
    q = raw[..., -128:].reshape(N, -1, 4, 32)
    q = np.stack([q & 15, q >> 4], 3).reshape(N, -1, n, 32).astype(np.int64)
    if t == GGMLType.Q5_K:
        q += (raw[..., 16:48].reshape(N, -1, 1, 32) >> np.arange(8).reshape(1, 1, 8, 1) & 1) << 4
    exact = q * (d.astype(np.float64)[..., None] * scale)[..., None] - (m.astype(np.float64)[..., None] * least)[..., None]
    return DeviceWeight.from_raw(raw.reshape(N, -1), t, (N, K), DEV), torch.from_numpy(exact.reshape(N, K)).to(DEV)


@pytest.mark.parametrize("t", [GGMLType.Q4_K, GGMLType.Q5_K])
@pytest.mark.parametrize("T", [16, 32, 64])
def test_few_tokens_see_the_rounded_weights(t, T):
    """One-hot tokens read the fp16 weights that the tensor cores get: scale q - min in fp32, rounded to fp16 once - also where scale and min are far apart."""
    N, K = 256, 512
    w, exact = _blocks(t, N, K, T)
    want = ops.dequant_rows(w, None, out=torch.empty(N, K, dtype=torch.float16, device=DEV))
    assert nmse(exact, want) < 1e-7
    eye = torch.eye(K, device=DEV, dtype=torch.float16)
    got = torch.cat([ops.linear(w, eye[i:i + T].contiguous(), "f32") for i in range(0, K, T)])
    assert torch.equal(got, want.float().T)


@pytest.mark.parametrize("t", [GGMLType.Q4_K, GGMLType.Q5_K])
@pytest.mark.parametrize("T", [1, 2, 4])
def test_mat_vec_on_mins_is_fp32(t, T):
    """Activations that 8 bits hold exactly (whole numbers, 127 the largest of 32): what remains is fp32 arithmetic.  Every 32 columns add a product of
    rounded scale, sum and offset - some 5 roundings of 2^-24 / sqrt(3) of terms as large as |scale q x| + |min x| together, added up at random."""
    N, K = 512, 4096
    w, exact = _blocks(t, N, K, 7)
    g = torch.Generator(DEV).manual_seed(T)
    x = torch.randint(-126, 127, (T, K), device=DEV, generator=g)
    x[:, ::32] = 127
    y = ops.linear(w, x.half(), "f32")
    ref = x.double() @ exact.T
    size = (x.double().abs()[:, None] * exact.abs()[None]).view(T, N, -1, 32).sum(-1).pow(2).sum(-1).sqrt()
    err = float(((y.double() - ref) / size).pow(2).mean().sqrt()) * 2 ** 24
    print("error / 2^-24:", err)
    assert err < 5 ** 0.5 / 3 ** 0.5


@pytest.mark.parametrize("t", [GGMLType.Q8_0, GGMLType.Q4_K, GGMLType.Q5_K, GGMLType.Q6_K])
@pytest.mark.parametrize("T,N,K,kib", [(193, 256, 256, 256), (300, 700, 512, 512), (1025, 1280, 768, 1 << 16)])
def test_linear_quant_prompt_in_pieces(t, T, N, K, kib):
    """Prompts on block types: one row tile a piece, pieces of which the last is partial, the whole matrix at once; bounds as for few tokens."""
    w, exact = _w(N, K, t, 1)
    u, exact_u = _w(N, K, t, 2)
    x = torch.randn(T, K, device=DEV, generator=torch.Generator(DEV).manual_seed(3)).half()
    ref = x.double() @ exact.double().T
    scratch = torch.empty(kib << 10, dtype=torch.uint8, device=DEV)
    assert nmse(ref, ops.linear(w, x, "f32", scratch=scratch)) < 2e-7 and nmse(ref, ops.linear(w, x, "f32")) < 2e-7
    acc = torch.ones(T, N, device=DEV)
    assert nmse(ref + 1, ops.linear(w, x, "add", out=acc, scratch=scratch)) < 2e-7
    assert nmse(torch.nn.functional.silu(ref) * (x.double() @ exact_u.double().T), ops.linear(w, x, "swiglu", w_up=u)) < 2e-6


def test_linear_quant_two_pass_scratch_entry_point():
    """dlp_linear's caller-provided-scratch contract still holds (used when DLP_GEMM_DEQUANT_SCRATCH=1)."""
    import ctypes as C
    from distributed_llm_pipeline_b200.ops import lib as L
    T, N, K = 48, 256, 512
    w, exact = _w(N, K, GGMLType.Q8_0, 4)
    x = torch.randn(T, K, device=DEV).half()
    y = torch.empty(T, N, device=DEV)
    scratch = torch.empty(N * K * 2, dtype=torch.uint8, device=DEV)
    rc = L.load().dlp_linear(w.ref(), None, x.data_ptr(), None, 0.0, y.data_ptr(), N, 1, T, scratch.data_ptr(), scratch.numel(),
                             torch.cuda.current_stream().cuda_stream)
    assert rc == 0 and nmse(x.float() @ exact.T, y) < 5e-6


def test_prompt_without_room_for_pieces(monkeypatch):
    """More than 192 tokens on block types where nothing can be allocated: the weights are unpacked in the GEMM instead."""
    w, exact = _w(512, 1024, GGMLType.Q4_K, 1)
    x = torch.randn(300, 1024, device=DEV, generator=torch.Generator(DEV).manual_seed(3)).half()
    out, empty = torch.empty(300, 512, device=DEV), torch.empty

    def full(*a, dtype=None, **kw):
        if dtype == torch.uint8:
            raise torch.OutOfMemoryError("no room")
        return empty(*a, dtype=dtype, **kw)
    monkeypatch.setattr(torch, "empty", full)
    ops.linear(w, x, "f32", out=out)
    assert nmse(x.double() @ exact.double().T, out) < 2e-7


def test_products_with_an_operand_unpacked_just_before():
    """Rows unpacked by one launch are the weights of the next, which may be requested early only where nothing writes them: different weights through
    one buffer, back to back, against 64 bits (fp16 values, fp32 sums)."""
    N, K, T = 384, 2048, (3, 5, 16, 17, 64, 65, 300)
    ws = [_w(N, K, t, i) for i, t in enumerate((GGMLType.Q8_0, GGMLType.Q4_K, GGMLType.Q6_K))]
    buf = torch.full((N, K), math.nan, dtype=torch.float16, device=DEV)
    xs = [torch.randn(t, K, device=DEV, generator=torch.Generator(DEV).manual_seed(t)).half() for t in T]
    cases = [(x, w, x.double() @ exact.half().double().T, torch.zeros(len(x), N, device=DEV)) for x in xs for _ in range(3) for w, exact in ws]
    for x, w, _, y in cases:
        ops.dequant_rows(w, None, out=buf)
        ops.gemm_f16(buf, x, y, epilogue=1)
    assert max(nmse(ref, y) for _, _, ref, y in cases) < 1e-11


_WHOLE_MATRIX_UNPACKED = """
import ctypes as C, sys, torch
sys.path.insert(0, "tests")
from test_kernels_gpu import _w, nmse, ops, GGMLType
from distributed_llm_pipeline_b200.ops import lib as L
assert ops.TWO_PASS_DEQUANT
N, K = 384, 1024
(a, ea), (b, eb) = _w(N, K, GGMLType.Q4_K, 1), _w(N, K, GGMLType.Q8_0, 2)
scratch = torch.full((N * K * 2,), float("nan"), dtype=torch.float16, device="cuda").view(torch.uint8)
for T in (3, 5, 16, 64, 100):
    x = torch.randn(T, K, device="cuda").half()
    ra, rb = x.double() @ ea.double().T, x.double() @ eb.double().T
    silu = torch.nn.functional.silu
    for _ in range(3):
        ys = []
        for w, u in ((a, None), (b, None), (b, b), (a, a)):
            y = torch.zeros(T, N, device="cuda", dtype=torch.float16 if u else torch.float32)
            rc = L.load().dlp_linear(w.ref(), u.ref() if u else None, x.data_ptr(), None, 0.0, y.data_ptr(), N, 3 if u else 1, T, scratch.data_ptr(), scratch.numel(),
                                     torch.cuda.current_stream().cuda_stream)
            assert rc == 0
            ys.append(y)
        for y, ref in zip(ys, (ra, rb, silu(rb) * rb, silu(ra) * ra)):
            assert nmse(ref, y) < 2e-6, T
print("ok")
"""


def test_whole_matrix_unpacked_to_scratch():
    """DLP_GEMM_DEQUANT_SCRATCH=1 (read once a process): weights that share one scratch, one call after the other, with and without a gate."""
    import os
    import subprocess
    import sys
    res = subprocess.run([sys.executable, "-c", _WHOLE_MATRIX_UNPACKED], capture_output=True, text=True, timeout=300, env={**os.environ, "DLP_GEMM_DEQUANT_SCRATCH": "1", "PYTHONPATH": "."})
    assert res.returncode == 0 and "ok" in res.stdout, res.stdout + res.stderr


def test_rmsnorm_with_residual():
    T, E = 7, 1024
    h = torch.randn(T, E, device=DEV)
    d = torch.randn(T, E, device=DEV)
    w = torch.rand(E, device=DEV) + 0.5
    ref_h = h + d
    ref = ref_h * torch.rsqrt(ref_h.pow(2).mean(-1, keepdim=True) + 1e-5) * w
    out = ops.rmsnorm(h, w, 1e-5, delta=d)
    assert torch.allclose(h, ref_h, atol=1e-6) and nmse(ref, out) < 1e-6


@pytest.mark.parametrize("affine", ["wb", "w", "none"])
@pytest.mark.parametrize("T,E", [(1, 256), (7, 1024), (130, 6144)])
def test_layernorm_with_residual(affine, T, E):
    """LayerNorm of the starcoder2 / falcon / olmo / orion / command-r families against torch in fp32: with weight and bias, weight
    only, and no parameters; the residual add into h included."""
    h = torch.randn(T, E, device=DEV) * 2 + 0.5          # non-zero mean: the centring matters
    d = torch.randn(T, E, device=DEV)
    w = (torch.rand(E, device=DEV) + 0.5) if affine != "none" else None
    b = torch.randn(E, device=DEV) * 0.1 if affine == "wb" else None
    ref_h = h + d
    ref = torch.nn.functional.layer_norm(ref_h, (E,), w, b, 1e-5)
    out = ops.layernorm(h, w, b, 1e-5, delta=d)
    assert torch.allclose(h, ref_h, atol=1e-6) and nmse(ref, out) < 1e-6
    h2 = ref_h.clone()
    assert nmse(ref, ops.layernorm(h2, w, b, 1e-5)) < 1e-6 and torch.equal(h2, ref_h)      # without delta h is left alone


@pytest.mark.parametrize("act", ["gelu", "gelu_erf", "relu2", "silu", "none"])
def test_bias_act(act):
    """Bias + activation between the two mat-muls of a non-gated MLP, against torch in fp32."""
    T, F = 9, 1536
    x = torch.randn(T, F, device=DEV) * 3
    bias = torch.randn(F, device=DEV)
    fn = {"none": lambda t: t, "gelu": lambda t: torch.nn.functional.gelu(t, approximate="tanh"), "relu2": lambda t: torch.relu(t) ** 2,
          "silu": torch.nn.functional.silu, "gelu_erf": torch.nn.functional.gelu}[act]
    assert nmse(fn(x + bias), ops.bias_act(x, bias, act)) < 1e-6
    assert nmse(fn(x), ops.bias_act(x, None, act)) < 1e-6


@pytest.mark.parametrize("neox", [False, True])
@pytest.mark.parametrize("D", [64, 128])
def test_rope_kv_write(neox, D):
    T, Hq, Hkv, page = 9, 4, 2, 16
    qkv = torch.randn(T, (Hq + 2 * Hkv) * D, device=DEV)
    pos = torch.arange(30, 30 + T, dtype=torch.int32, device=DEV)
    pages = torch.tensor([3, 1, 2], dtype=torch.int32)
    slot = (pages[(pos.cpu() // page).long()] * page + pos.cpu() % page).to(torch.int32).to(DEV)
    inv = (10000.0 ** (-torch.arange(0, D // 2).double() * 2 / D)).float().to(DEV)
    kc = torch.zeros(4, Hkv, page, D, dtype=torch.float16, device=DEV)
    vc = torch.zeros_like(kc)
    q = ops.rope_kv(qkv, pos, slot, inv, kc, vc, Hq, Hkv, D, neox)
    x = qkv.view(T, Hq + 2 * Hkv, D)
    q_ref = apply_rope(x[:, :Hq].cpu(), pos.cpu(), inv.cpu(), neox) / math.sqrt(D)
    k_ref = apply_rope(x[:, Hq:Hq + Hkv].cpu(), pos.cpu(), inv.cpu(), neox)
    assert nmse(q_ref.reshape(T, -1), q) < 1e-6
    pg, off = (slot.cpu() // page).long(), (slot.cpu() % page).long()
    assert nmse(k_ref, kc.cpu()[pg, :, off]) < 1e-6
    assert nmse(x[:, Hq + Hkv:].cpu(), vc.cpu()[pg, :, off]) < 1e-6


@pytest.mark.parametrize("in_dtype", [torch.float32, torch.float16])
@pytest.mark.parametrize("D,with_bias,with_norm", [(64, True, False), (128, False, True), (64, True, True), (128, True, True)])
def test_rope_kv_bias_and_head_norm(D, with_bias, with_norm, in_dtype):
    """qwen2 bias / qwen3 per-head Q,K RMSNorm fused into the RoPE + KV-write launch, against the fp32 formula."""
    from distributed_llm_pipeline_b200.models.reference import rms_norm
    T, Hq, Hkv, page, eps = 7, 6, 2, 16, 1e-6
    H = Hq + 2 * Hkv
    qkv = torch.randn(T, H * D, device=DEV).to(in_dtype)
    pos = torch.arange(3, 3 + T, dtype=torch.int32, device=DEV)
    slot = (pos + 2 * page).to(torch.int32)
    inv = (10000.0 ** (-torch.arange(0, D // 2).double() * 2 / D)).float().to(DEV)
    kc = torch.zeros(4, Hkv, page, D, dtype=torch.float16, device=DEV)
    vc = torch.zeros_like(kc)
    bias = torch.randn(H * D, device=DEV) * 0.3 if with_bias else None
    qn = 1 + 0.2 * torch.randn(D, device=DEV) if with_norm else None
    kn = 1 + 0.2 * torch.randn(D, device=DEV) if with_norm else None
    q = ops.rope_kv(qkv, pos, slot, inv, kc, vc, Hq, Hkv, D, True, bias=bias, q_norm=qn, k_norm=kn, eps=eps)
    x = qkv.float().cpu()
    if with_bias:
        x = x + bias.cpu()
    x = x.view(T, H, D)
    xq, xk = x[:, :Hq], x[:, Hq:Hq + Hkv]
    if with_norm:
        xq, xk = rms_norm(xq, qn.cpu(), eps), rms_norm(xk, kn.cpu(), eps)
    q_ref = apply_rope(xq, pos.cpu(), inv.cpu(), True) / math.sqrt(D)
    k_ref = apply_rope(xk, pos.cpu(), inv.cpu(), True)
    tol = 1e-6 if in_dtype == torch.float32 else 2e-6
    assert nmse(q_ref.reshape(T, -1), q) < tol
    pg, off = (slot.cpu() // page).long(), (slot.cpu() % page).long()
    assert nmse(k_ref, kc.cpu()[pg, :, off]) < tol
    assert nmse(x[:, Hq + Hkv:], vc.cpu()[pg, :, off]) < tol


def _fill_cache(n_pages, Hkv, page, D, seed=0):
    g = torch.Generator(device=DEV).manual_seed(seed)
    kc = torch.randn(n_pages, Hkv, page, D, device=DEV, generator=g).half()
    vc = torch.randn(n_pages, Hkv, page, D, device=DEV, generator=g).half()
    return kc, vc


@pytest.mark.parametrize("D,Hq,Hkv", [(128, 8, 2), (64, 8, 1), (128, 4, 4), (64, 6, 3)])
@pytest.mark.parametrize("n_splits", [1, 4])
def test_attn_paged_decode(D, Hq, Hkv, n_splits):
    page, n_pages, max_pages = 16, 200, 48
    kc, vc = _fill_cache(n_pages, Hkv, page, D)
    lens = torch.tensor([1, 17, 300, 700], dtype=torch.int32, device=DEV)   # short: single CTA; long: split-KV + combine
    nq = lens.numel()
    bt = torch.randperm(n_pages)[: nq * max_pages].view(nq, max_pages).to(torch.int32).to(DEV)
    q = (torch.randn(nq, Hq * D, device=DEV) / math.sqrt(D)).half()
    out = ops.attn_paged(q, kc, vc, bt, lens, Hq, Hkv, D, n_splits=n_splits)
    ref = ops._attn_cpu(q.cpu(), kc.cpu(), vc.cpu(), bt.cpu(), lens.cpu(), Hq, Hkv, D)
    assert nmse(ref, out) < 5e-5
    if n_splits > 1:   # combine fused into the attention kernel (last split CTA merges); twice: counters must self-reset
        ws = (torch.empty(nq * Hq * n_splits * D, device=DEV), torch.empty(nq * Hq * n_splits * 2, device=DEV),
              torch.zeros(nq * Hq, dtype=torch.int32, device=DEV))
        for _ in range(2):
            out2 = ops.attn_paged(q, kc, vc, bt, lens, Hq, Hkv, D, n_splits=n_splits, workspace=ws)
            assert nmse(ref, out2) < 5e-5
        assert int(ws[2].abs().sum()) == 0


@pytest.mark.parametrize("D,Hq,Hkv", [(128, 8, 2), (64, 8, 1), (128, 4, 4), (64, 6, 3)])
@pytest.mark.parametrize("neox", [False, True])
@pytest.mark.parametrize("n_splits", [1, 8, 16])
def test_attn_decode_rope_onepass(D, Hq, Hkv, neox, n_splits):
    """RoPE + K/V page write + split-KV attention + cluster (DSMEM) combine in one launch, against the separate fp32 steps."""
    page, n_pages, max_pages = 16, 400, 80
    kc, vc = _fill_cache(n_pages, Hkv, page, D, seed=3)
    lens = torch.tensor([1, 2, 17, 64, 65, 300, 700, 1200], dtype=torch.int32, device=DEV)   # kv_len includes the new token
    nq = lens.numel()
    bt = torch.randperm(n_pages)[: nq * 40].view(nq, 40).to(torch.int32)
    bt = torch.cat([bt, torch.zeros(nq, max_pages - 40, dtype=torch.int32)], 1).to(DEV)          # 8 x 40 pages of 16 = 640 < 1200?
    lens = torch.minimum(lens, torch.tensor(40 * page, device=DEV)).to(torch.int32)
    H = Hq + 2 * Hkv
    qkv = torch.randn(nq, H * D, device=DEV)
    inv = (10000.0 ** (-torch.arange(0, D // 2).double() * 2 / D)).float().to(DEV)
    # oracle: CPU rope + cache write + attention on copies of the cache
    kc_ref, vc_ref = kc.cpu().clone(), vc.cpu().clone()
    pos = (lens - 1).cpu()
    slot = (bt.cpu()[torch.arange(nq), (pos // page).long()] * page + pos % page).to(torch.int32)
    q_ref = ops.rope_kv(qkv.cpu(), pos.to(torch.int32), slot, inv.cpu(), kc_ref, vc_ref, Hq, Hkv, D, neox)
    ref = ops._attn_cpu(q_ref, kc_ref, vc_ref, bt.cpu(), lens.cpu(), Hq, Hkv, D)
    ang = pos.float()[:, None] * inv.cpu()[None]
    table = torch.stack([ang.cos(), ang.sin()], -1).contiguous().to(DEV)      # the per-step table advance_rope writes
    for tab in (None, table):      # in-kernel sincos, then the table; the second call rewrites the same slots with the same values
        out = ops.attn_decode_rope(qkv, inv, kc, vc, bt, lens, Hq, Hkv, D, n_splits=n_splits, neox=neox, rope_cs=tab)
        assert nmse(ref, out) < 5e-5
    pg, off = (slot // page).long(), (slot % page).long()
    assert nmse(kc_ref[pg, :, off], kc.cpu()[pg, :, off]) < 1e-6
    assert nmse(vc_ref[pg, :, off], vc.cpu()[pg, :, off]) < 1e-6
    untouched = torch.ones(n_pages, dtype=torch.bool)
    untouched[pg] = False
    assert torch.equal(kc.cpu()[untouched], kc_ref[untouched])          # nothing else in the cache was written


@pytest.mark.parametrize("D,Hq,Hkv", [(128, 8, 2), (64, 16, 2), (128, 24, 2), (64, 40, 2)])      # 4, 8, 12 and 20 query heads to a key head
@pytest.mark.parametrize("page", [16, 64])
@pytest.mark.parametrize("n_splits", [1, 3, 40])
def test_attn_split_tiles_and_joins(D, Hq, Hkv, page, n_splits):
    """Split-KV attention at the edges of its tiles (16 keys), warps (4 tiles) and splits (256 keys), with and without RoPE and the new token's
    K / V in the same launch, against 64 bits.  Bound: the output is rounded to fp16 (relative 2^-12 on average, squared 6e-8)."""
    lens = [1, 15, 16, 17, 64, 65, 256, 257, 511, 513, 1040, 3001]
    nq, per = len(lens), (max(lens) + page - 1) // page
    kc, vc = _fill_cache(nq * per, Hkv, page, D, seed=5)
    bt = torch.randperm(nq * per, generator=torch.Generator().manual_seed(1)).view(nq, per).to(torch.int32).to(DEV)
    kv_len = torch.tensor(lens, dtype=torch.int32, device=DEV)
    qkv = torch.randn(nq, (Hq + 2 * Hkv) * D, device=DEV, generator=torch.Generator(DEV).manual_seed(2))
    inv = (10000.0 ** (-torch.arange(0, D // 2).double() * 2 / D)).float().to(DEV)
    ws = (torch.full((nq * Hq * n_splits * D,), math.nan, device=DEV), torch.full((nq * Hq * n_splits * 2,), math.nan, device=DEV),
          torch.zeros(nq * Hq, dtype=torch.int32, device=DEV))

    def exact(q, i, n):
        pg = bt[i, :(n + page - 1) // page].long()
        k, v = (c[pg].permute(1, 0, 2, 3).reshape(Hkv, -1, D)[:, :n].double().repeat_interleave(Hq // Hkv, 0) for c in (kc, vc))
        return (torch.softmax(k @ q.view(Hq, D, 1).double(), 1) * v).sum(1).view(-1)
    for neox in (False, True):
        out = ops.attn_decode_rope(qkv, inv, kc, vc, bt, kv_len, Hq, Hkv, D, n_splits=n_splits, neox=neox, workspace=ws)
        x = qkv.double().view(nq, -1, D)
        for i, n in enumerate(lens):
            a = (n - 1) * inv.double()
            rot = x[i, :Hq + Hkv]
            u, v = (rot[:, :D // 2], rot[:, D // 2:]) if neox else (rot[:, 0::2], rot[:, 1::2])
            pair = (u * a.cos() - v * a.sin(), u * a.sin() + v * a.cos())
            rot = torch.cat(pair, -1) if neox else torch.stack(pair, -1).flatten(-2)
            row = (bt[i, (n - 1) // page].long(), slice(None), (n - 1) % page)
            assert nmse(rot[Hq:], kc[row]) < 1e-6 and torch.equal(x[i, Hq + Hkv:].half(), vc[row])
            assert nmse(exact(rot[:Hq] * D ** -0.5, i, n), out[i]) < 2e-7, (neox, n)
    q = (torch.randn(nq, Hq * D, device=DEV) / math.sqrt(D)).half()
    joined = ops.attn_paged(q, kc, vc, bt, kv_len, Hq, Hkv, D, n_splits=n_splits, workspace=ws)
    assert torch.equal(joined, ops.attn_paged(q, kc, vc, bt, kv_len, Hq, Hkv, D, n_splits=n_splits))
    for i, n in enumerate(lens):
        assert nmse(exact(q[i], i, n), joined[i]) < 2e-7, n
    assert int(ws[2].abs().sum()) == 0


@pytest.mark.parametrize("lens", [[300] * 31 + [9000], [20, 7000, 330], [321, 320, 0, 1], [2000] * 16, [100 * i for i in range(40)], [5] * 70 + [3000] + [400] * 29, [65] * 290 + [700] * 10])
@pytest.mark.parametrize("n_splits", [2, 5])
def test_attn_split_of_uneven_batches(lens, n_splits):
    """Queries that share a pool of key ranges: one long among short ones, empty ones, more than a warp of queries, more than share (256), pools that are too small
    for short ranges.  Joined in the kernel and by a second one, against 64 bits; a long one beside short ones takes most of the pool."""
    D, Hq, Hkv, page, nq = 64, 8, 2, 64, len(lens)
    need = [(n + page - 1) // page for n in lens]
    kc, vc = _fill_cache(sum(need) + 1, Hkv, page, D, seed=5)
    bt = torch.zeros(nq, max(need), dtype=torch.int32)
    for i, n in enumerate(need):
        bt[i, :n] = torch.arange(n) + sum(need[:i])
    bt, kv_len = bt.to(DEV), torch.tensor(lens, dtype=torch.int32, device=DEV)
    q = (torch.randn(nq, Hq * D, device=DEV, generator=torch.Generator(DEV).manual_seed(1)) / math.sqrt(D)).half()
    ws = (torch.full((nq * Hq * n_splits * D,), math.nan, device=DEV), torch.full((nq * Hq * n_splits * 2,), math.nan, device=DEV), torch.zeros(nq * Hq, dtype=torch.int32, device=DEV))
    out = ops.attn_paged(q, kc, vc, bt, kv_len, Hq, Hkv, D, n_splits=n_splits, workspace=ws)
    assert torch.equal(out, ops.attn_paged(q, kc, vc, bt, kv_len, Hq, Hkv, D, n_splits=n_splits))
    assert int(ws[2].abs().sum()) == 0
    for i, n in enumerate(lens):
        if n == 0:
            assert not out[i].any()
            continue
        pg = bt[i, :need[i]].long()
        k, v = (c[pg].permute(1, 0, 2, 3).reshape(Hkv, -1, D)[:, :n].double().repeat_interleave(Hq // Hkv, 0) for c in (kc, vc))
        ref = (torch.softmax(k @ q[i].view(Hq, D, 1).double(), 1) * v).sum(1).view(-1)
        assert nmse(ref, out[i]) < 2e-7, (i, n)
    if lens[-1] == 9000:
        ranges = int((~ws[1].view(Hq, -1, 2)[0, :, 0].isnan()).sum())
        assert ranges >= 16


@pytest.mark.parametrize("D,Hq,Hkv", [(128, 32, 8), (64, 32, 4), (128, 24, 2)])
def test_attn_split_arithmetic_is_fp32(D, Hq, Hkv):
    """Sums that cancel show what decode attention rounds: keys with values + 1024, others, and the first keys again with - 1024.  Each rounding of an fp32 sum of
    that size is 2^-24 / sqrt(3) of it (rms); kept in the tensor cores' sums, which cut off, the error was 0.9 to 1.0 of 2^-24."""
    page, n, err = 64, 300, {}
    for rope in (False, True):
        for seed in range(4):
            g = torch.Generator(DEV).manual_seed(seed)
            T = 3 * n
            per = (T + page) // page
            k, other = ((torch.randn(Hkv, n, D, device=DEV, generator=g) * 0.3) for _ in range(2))
            big = torch.full((Hkv, n, D), 1024.0, device=DEV)
            K = torch.cat([k, other, k], 1).half()
            V = torch.cat([big, torch.randn(Hkv, n, D, device=DEV, generator=g), -big], 1).half()
            kc, vc = torch.zeros(2, per, Hkv, page, D, device=DEV, dtype=torch.float16)
            for cache, rows in ((kc, K), (vc, V)):
                flat = torch.zeros(Hkv, per * page, D, device=DEV, dtype=torch.float16)
                flat[:, :T] = rows
                cache.copy_(flat.view(Hkv, per, page, D).permute(1, 0, 2, 3))
            bt = torch.arange(per, dtype=torch.int32, device=DEV)[None].contiguous()
            ws = (torch.zeros(Hq * 16 * D, device=DEV), torch.zeros(Hq * 32, device=DEV), torch.zeros(Hq, dtype=torch.int32, device=DEV))
            if rope:            # (angles 0; the new token's own value is 0)
                qkv = torch.randn(1, (Hq + 2 * Hkv) * D, device=DEV, generator=g)
                qkv[:, (Hq + Hkv) * D:] = 0
                out = ops.attn_decode_rope(qkv, torch.zeros(D // 2, device=DEV), kc, vc, bt, torch.tensor([T + 1], dtype=torch.int32, device=DEV), Hq, Hkv, D, n_splits=16, workspace=ws)
                q = qkv.double().view(-1, D)[:Hq] * torch.tensor(D ** -0.5, dtype=torch.float32).double().item()
                K, V = torch.cat([K, qkv.view(-1, D)[Hq:Hq + Hkv, None].half()], 1), torch.cat([V, torch.zeros_like(V[:, :1])], 1)
            else:
                q = (torch.randn(1, Hq * D, device=DEV, generator=g) * D ** -0.5).half()
                out = ops.attn_paged(q, kc, vc, bt, torch.tensor([T], dtype=torch.int32, device=DEV), Hq, Hkv, D, n_splits=16, workspace=ws)
                q = q.double().view(Hq, D)
            p = torch.softmax(torch.einsum("hd,hnd->hn", q, K.double().repeat_interleave(Hq // Hkv, 0)), -1)
            V = V.double().repeat_interleave(Hq // Hkv, 0)
            e = (out.double().view(Hq, D) - torch.einsum("hn,hnd->hd", p, V)) / torch.einsum("hn,hnd->hd", p, V.abs())
            err.setdefault(rope, []).append(float(e.pow(2).mean().sqrt()) * 2 ** 24)
    assert all(sum(v) / len(v) < 3 ** -0.5 for v in err.values()), err


@pytest.mark.parametrize("size", [1e-12, 3e5, 1e9])
def test_attn_split_takes_queries_of_any_size(size):
    """fp32 queries beyond what fp16 holds, up and down, against keys of the inverse size: the scores are ordinary."""
    D, Hq, Hkv, page, n = 128, 8, 2, 16, 200
    kc, vc = _fill_cache(16, Hkv, page, D, seed=3)
    kc = (kc.float() * max(min(1 / size, 1e3), 2e-5)).half()
    scale = size * float(kc.float().std())
    qkv = torch.randn(1, (Hq + 2 * Hkv) * D, device=DEV, generator=torch.Generator(DEV).manual_seed(2)) * size
    qkv[:, Hq * D:] = 0.5
    ws = (torch.zeros(Hq * 4 * D, device=DEV), torch.zeros(Hq * 8, device=DEV), torch.zeros(Hq, dtype=torch.int32, device=DEV))
    bt = torch.arange(16, dtype=torch.int32, device=DEV)[None].contiguous()
    out = ops.attn_decode_rope(qkv, torch.zeros(D // 2, device=DEV), kc, vc, bt, torch.tensor([n], dtype=torch.int32, device=DEV), Hq, Hkv, D, n_splits=4, workspace=ws,
                               attn_scale=1 / scale)
    k, v = (c.permute(1, 0, 2, 3).reshape(Hkv, -1, D)[:, :n].double().repeat_interleave(Hq // Hkv, 0) for c in (kc, vc))
    q = qkv.double().view(-1, D)[:Hq] * (D ** -0.5 / scale)
    ref = torch.einsum("hn,hnd->hd", torch.softmax(torch.einsum("hd,hnd->hn", q, k), -1), v)
    assert nmse(ref.view(1, -1), out) < 2e-7


@pytest.mark.parametrize("impl", ["tc", "mma"])
@pytest.mark.parametrize("D,Hq,Hkv", [(128, 8, 2), (64, 4, 2)])
@pytest.mark.parametrize("T,pos0,page", [(5, 0, 16), (64, 0, 16), (100, 37, 16), (200, 64, 16), (128, 0, 64), (300, 250, 64), (513, 1000, 64), (1, 400, 8)])
def test_attn_prefill_causal(D, Hq, Hkv, T, pos0, page, impl):
    """Both prefill-attention kernels (tcgen05/TMEM/TMA and the mma.sync FA-2 one) against fp32 attention over the same pages:
    tiles that end inside a page, chunks that start mid-sequence, more than one 128-query tile, several 128-key tiles."""
    total = pos0 + T
    n_need = (total + page - 1) // page
    kc, vc = _fill_cache(n_need + 3, Hkv, page, D, seed=1)
    row = torch.randperm(n_need + 3)[:n_need].to(torch.int32).to(DEV)
    q = (torch.randn(T, Hq * D, device=DEV) / math.sqrt(D)).half()
    out = ops.attn_prefill(q, kc, vc, row, pos0, Hq, Hkv, D, impl=impl)
    kv_len = torch.arange(pos0 + 1, pos0 + T + 1, dtype=torch.int32)
    ref = ops._attn_cpu(q.cpu(), kc.cpu(), vc.cpu(), row.cpu().view(1, -1).expand(T, -1), kv_len, Hq, Hkv, D)
    assert nmse(ref, out) < 5e-4


@pytest.mark.parametrize("D,Hq,Hkv", [(128, 80, 8), (64, 72, 24), (64, 128, 128)])      # tiles of two heads; of 256 queries (3 and 1 heads to a key head)
@pytest.mark.parametrize("T,pos0,page", [(257, 0, 64), (300, 129, 16), (384, 1000, 128), (520, 1, 32)])
def test_attn_prefill_two_tiles(D, Hq, Hkv, T, pos0, page):
    """Flash-prefill with two query tiles a block: last tiles of one row and a second tile that is not there, several key tiles, keys that end
    inside a page, scores that grow by more than 2^8 on the way (the output is rescaled).  Against 64 bits; the weights and the output are fp16."""
    n_need = (pos0 + T + page - 1) // page
    kc, vc = _fill_cache(n_need + 3, Hkv, page, D, seed=1)
    kc *= torch.linspace(0.2, 4, n_need + 3, device=DEV).view(-1, 1, 1, 1).to(kc.dtype)
    row = torch.arange(n_need).to(torch.int32).to(DEV)
    q = (torch.randn(T, Hq * D, device=DEV, generator=torch.Generator(DEV).manual_seed(4)) / math.sqrt(D)).half()
    out = ops.attn_prefill(q, kc, vc, row, pos0, Hq, Hkv, D)
    k, v = (c[row.long()].permute(1, 0, 2, 3).reshape(Hkv, -1, D)[:, :pos0 + T].double() for c in (kc, vc))
    hidden = torch.arange(pos0 + T, device=DEV)[None] > pos0 + torch.arange(T, device=DEV)[:, None]
    ref = torch.empty(T, Hq, D, dtype=torch.float64, device=DEV)
    for h in range(Hq):
        s = (q.view(T, Hq, D)[:, h].double() @ k[h * Hkv // Hq].T).masked_fill(hidden, -math.inf)
        ref[:, h] = torch.softmax(s, -1) @ v[h * Hkv // Hq]
    assert nmse(ref.view(T, -1), out) < 3e-7


def test_argmax_and_sampler():
    R, V = 3, 32000
    lg = torch.randn(R, V, device=DEV)
    assert torch.equal(ops.argmax(lg).long(), lg.argmax(-1))
    # greedy through the sampler entry point
    assert torch.equal(ops.sample(lg, temp=0.0).long(), lg.argmax(-1))
    # top_k=1 must return the argmax whatever the temperature
    assert torch.equal(ops.sample(lg, top_k=1, temp=1.5).long(), lg.argmax(-1))
    # draws stay inside the top-k set and follow the distribution roughly
    lg2 = torch.full((1, V), -10.0, device=DEV)
    lg2[0, 7], lg2[0, 99], lg2[0, 1234] = 2.0, 1.0, 0.0
    ctr = torch.zeros(1, dtype=torch.int32, device=DEV)
    counts = {7: 0, 99: 0, 1234: 0}
    for i in range(300):
        ctr.fill_(i)
        t = int(ops.sample(lg2, top_k=3, top_p=1.0, min_p=0.0, temp=1.0, seed=5, step_ctr=ctr)[0])
        assert t in counts
        counts[t] += 1
    assert counts[7] > counts[99] > counts[1234] > 0
    # top-p keeps only the head of the distribution
    for i in range(50):
        ctr.fill_(i)
        assert int(ops.sample(lg2, top_k=40, top_p=0.5, min_p=0.0, temp=1.0, seed=1, step_ctr=ctr)[0]) == 7


def test_advance_bookkeeping():
    page, B, max_pages = 16, 3, 4
    bt = torch.arange(B * max_pages, dtype=torch.int32, device=DEV).view(B, max_pages)
    sl = torch.tensor([0, 15, 16], dtype=torch.int32, device=DEV)
    pos = torch.zeros(B, dtype=torch.int32, device=DEV)
    slot = torch.zeros(B, dtype=torch.int32, device=DEV)
    kvl = torch.zeros(B, dtype=torch.int32, device=DEV)
    ops.advance(sl, None, pos, slot, kvl, bt, page, B)
    assert kvl.tolist() == [1, 16, 17]
    assert pos.tolist() == [0, 15, 16] and sl.tolist() == [1, 16, 17]
    assert slot.tolist() == [0 * 16 + 0, 4 * 16 + 15, 9 * 16 + 0]


@pytest.mark.parametrize("t", [GGMLType.F16, GGMLType.Q8_0, GGMLType.Q4_K])
@pytest.mark.parametrize("T", [1, 2, 4])
def test_fused_allreduce_protocol_virtual_ranks(t, T):
    """Row-parallel GEMV -> self-signalling stores into every rank's buffer; next GEMV's prologue spins on the values, folds
    h += sum(partials) into its RMSNorm and re-arms the other parity.  Four virtual ranks on one GPU, phases launched rank by
    rank (no co-scheduled waiting kernels); five steps so that both parities are reused after being re-armed."""
    from distributed_llm_pipeline_b200.parallel.fused import FusedComm
    tp, E, F = 4, 512, 1024
    comms = FusedComm.make_virtual(tp, E, n_sites=2)
    g = torch.Generator().manual_seed(11)
    w_down = torch.randn(E, F, generator=g) * 0.05          # row-parallel: K = F sharded
    w_next = torch.randn(256, E, generator=g) * 0.05         # next column-parallel matrix (replicated here)
    nw = (torch.rand(E, generator=g) + 0.5).to(DEV)
    act = (torch.randn(T, F, generator=g)).half().to(DEV)
    h = torch.randn(T, E, generator=g).to(DEV)
    Fs = F // tp
    shards = [DeviceWeight.from_dense(w_down[:, r * Fs:(r + 1) * Fs].contiguous(), t, DEV) for r in range(tp)]
    wn = DeviceWeight.from_dense(w_next, t, DEV)
    from distributed_llm_pipeline_b200.gguf.quants import dequantize, quantize
    import numpy as np
    deq = lambda m: torch.from_numpy(dequantize(quantize(m.numpy(), t), t, tuple(m.shape)).astype(np.float32)).to(DEV)
    for step in range(5):                                       # several epochs through the same site: no stale data
        for c in comms:
            c.begin_step()
        for r, c in enumerate(comms):                           # phase 1: every rank pushes its partial rows
            c.gemv(shards[r], act[:, r * Fs:(r + 1) * Fs].contiguous(), 4, T, ar_out=c.ar_out(0))
        partial_sum = sum(act[:, r * Fs:(r + 1) * Fs].float() @ deq(w_down[:, r * Fs:(r + 1) * Fs].contiguous()).T for r in range(tp))
        h_ref = h + partial_sum
        xn = (h_ref * torch.rsqrt(h_ref.pow(2).mean(-1, keepdim=True) + 1e-5) * nw).half().float()
        y_ref = xn @ deq(w_next).T
        for r, c in enumerate(comms):                           # phase 2: every rank consumes
            h_out = torch.zeros_like(h)
            y = torch.empty(T, 256, device=DEV)
            c.gemv(wn, h, 1, T, out=y, norm_w=nw, eps=1e-5, ar_in=c.ar_in(0, h_out))
            assert nmse(h_ref, h_out) < (1e-4 if t.name.startswith("Q") else 1e-6)
            assert nmse(y_ref, y) < (3e-4 if t.name.startswith("Q") else 2e-5)
            c.check_error()
        act = (act.float() * 0.5 + 0.1).half()


def test_fused_allreduce_passes_negative_zero_and_changing_batch():
    """-0.0 is the "empty" pattern on the wire: a partial that is exactly -0.0 must arrive as +0.0, not hang the consumer; and a
    step with fewer token rows after one with more must not see the stale rows (the whole site is re-armed)."""
    from distributed_llm_pipeline_b200.parallel.fused import FusedComm
    tp, E, F = 2, 256, 512
    comms = FusedComm.make_virtual(tp, E, n_sites=1)
    g = torch.Generator().manual_seed(5)
    w_next = DeviceWeight.from_dense(torch.randn(64, E, generator=g) * 0.05, GGMLType.F16, DEV)
    nw = torch.ones(E, device=DEV)
    zero_w = [DeviceWeight.from_dense(torch.zeros(E, F // tp), GGMLType.F16, DEV) for _ in range(tp)]
    for step, T in enumerate([4, 1, 4, 2, 1]):
        act = -torch.ones(T, F // tp, dtype=torch.float16, device=DEV)       # (-1) * (+0) = -0.0 in every partial
        h = torch.randn(T, E, generator=g).to(DEV)
        for c in comms:
            c.begin_step()
        for r, c in enumerate(comms):
            c.gemv(zero_w[r], act, 4, T, ar_out=c.ar_out(0))
        for c in comms:
            h_out = torch.zeros_like(h)
            y = torch.empty(T, 64, device=DEV)
            c.gemv(w_next, h, 1, T, out=y, norm_w=nw, eps=1e-5, ar_in=c.ar_in(0, h_out))
            torch.cuda.synchronize()
            c.check_error()
            assert torch.equal(h_out, h), step


def test_sharded_argmax_emulated_rank():
    """dlp_argmax_tp on the single-device emulation (rank 0's stores land in every slot of its own buffer): picks the shard's
    best entry, lowest id on ties, offset by the shard's first global id; slots are re-armed across steps."""
    from distributed_llm_pipeline_b200.parallel.fused import FusedComm
    c = FusedComm.make_emulated(4, 256, 1)
    g = torch.Generator().manual_seed(9)
    for step in range(5):
        B, V, v0 = [1, 2, 4, 1, 37][step], 4099, 1000
        lg = torch.randn(B, V, generator=g).to(DEV)
        lg[0, 77] = lg[0, 300] = 50.0                      # tie: the lower id wins
        out = torch.zeros(B, dtype=torch.int32, device=DEV)
        c.argmax_sharded(lg, v0, out)
        torch.cuda.synchronize()
        c.check_error()
        want = lg.argmax(-1) + v0
        want[0] = 77 + v0
        assert out.tolist() == want.tolist(), step


def test_emulated_tp_engine_fused_equals_unfused(tmp_models):
    """The single-device emulation of a tp-way rank (bench.py --emulate-tp): its fused decode step (stores + spin + sharded
    arg-max inside a CUDA graph) must reproduce the unfused step of the same shard (separate all-reduce stand-in)."""
    from distributed_llm_pipeline_b200.models.llama import LlamaEngine
    from distributed_llm_pipeline_b200.models.weights import load_weights
    from distributed_llm_pipeline_b200.parallel.fused import FusedComm
    path = tmp_models[("tiny128", "F16")]
    tp = 2
    w = load_weights(path, "cuda", tp_rank=0, tp_size=tp)
    fused = LlamaEngine(w, n_ctx=128, max_seqs=2, page_size=16, max_batch_tokens=32, comm=FusedComm.make_emulated(tp))
    plain_comm = FusedComm.make_emulated(tp)
    plain_comm.fused = False
    plain = LlamaEngine(w, n_ctx=128, max_seqs=2, page_size=16, max_batch_tokens=32, comm=plain_comm)
    assert fused.fused_tp and not plain.fused_tp
    prompt = [1, 5, 9, 200, 33, 7, 8]
    sa, sb = fused.alloc_seq(), plain.alloc_seq()
    la, lb = fused.prefill(sa, prompt), plain.prefill(sb, prompt)
    assert nmse(lb, la) < 1e-5
    tok = int(lb.argmax())
    want = [tok]
    for _ in range(9):
        lb = plain.decode([sb], [want[-1]], sample=False, use_graph=False)[0]
        la = fused.decode([sa], [want[-1]], sample=False)[0]
        assert nmse(lb, la) < 1e-4
        want.append(int(lb.argmax()))
    fused.free_seq(sa)
    assert fused.generate(prompt, 10) == want            # device-fed tokens through the sharded arg-max
    fused.comm.check_error()


@pytest.mark.parametrize("t", [GGMLType.F16, GGMLType.Q8_0])
@pytest.mark.parametrize("T", [64, 200])
def test_fused_gemm_reduce_scatter_allgather_virtual_ranks(t, T):
    """Sequence-parallel prefill pair on 4 virtual ranks (one GPU, phases launched rank by rank):
    row-parallel GEMM --RS push--> owners' reduce buffers --rs_norm_ag--> everyone's gather buffer --AG wait--> GEMM."""
    from distributed_llm_pipeline_b200.parallel.fused import FusedComm
    from distributed_llm_pipeline_b200.gguf.quants import dequantize, quantize
    import numpy as np
    tp, E, F, N2 = 4, 512, 1024, 384
    Tp = (T + tp - 1) // tp * tp
    rows = Tp // tp
    comms = FusedComm.make_virtual_sp(tp, E, Tp)
    g = torch.Generator().manual_seed(21)
    w_down = torch.randn(E, F, generator=g) * 0.05
    w_next = torch.randn(N2, E, generator=g) * 0.05
    nw = (torch.rand(E, generator=g) + 0.5).to(DEV)
    act = torch.zeros(Tp, F)
    act[:T] = torch.randn(T, F, generator=g)
    act = act.half().to(DEV)
    h_full = torch.zeros(Tp, E)
    h_full[:T] = torch.randn(T, E, generator=g)
    h_full = h_full.to(DEV)
    Fs = F // tp
    deq = lambda m: torch.from_numpy(dequantize(quantize(m.numpy(), t), t, tuple(m.shape)).astype(np.float32)).to(DEV)
    shards = [DeviceWeight.from_dense(w_down[:, r * Fs:(r + 1) * Fs].contiguous(), t, DEV) for r in range(tp)]
    wn = DeviceWeight.from_dense(w_next, t, DEV)
    h_sh = [h_full[r * rows:(r + 1) * rows].clone() for r in range(tp)]
    for rep in range(2):        # twice through the same buffers: epochs advance, nothing stale is read
        for r, c in enumerate(comms):      # phase 1: row-parallel GEMM, partial tiles pushed to the owner ranks
            c.sp_gemm(shards[r], act[:, r * Fs:(r + 1) * Fs].contiguous(), Fs, Tp, rows, 5, rs_to=0)
        for r, c in enumerate(comms):      # phase 2: owners reduce + norm + push their rows into every gather buffer
            c.sp_norm_ag(h_sh[r], rows, nw, 1e-5, g=0, red=0)
        partial = sum(act[:, r * Fs:(r + 1) * Fs].float() @ deq(w_down[:, r * Fs:(r + 1) * Fs].contiguous()).T for r in range(tp))
        h_full = h_full + partial
        xn = (h_full * torch.rsqrt(h_full.pow(2).mean(-1, keepdim=True) + 1e-5) * nw).half().float()
        y_ref = xn @ deq(w_next).T
        for r, c in enumerate(comms):      # phase 3: column-parallel GEMM reads the gathered X (waits per owner flag)
            assert nmse(h_full[r * rows:(r + 1) * rows], h_sh[r]) < 1e-6
            y = torch.empty(Tp, N2, device=DEV)
            c.sp_gemm(wn, c.sp_gather_view(0, Tp), E, Tp, rows, 1, y=y, x_from_g=0)
            assert nmse(y_ref[:T], y[:T]) < 2e-5
            c.check_error()
        act = (act.float() * 0.7).half()


@pytest.mark.parametrize("t", [GGMLType.F16, GGMLType.Q8_0, GGMLType.Q4_K])
def test_moe_route_and_expert_indexed_gemv(t):
    """Device-side MoE decode pieces: router (softmax -> top-2 -> renormalise) and mat-vecs that pick the expert's rows
    from a stacked weight through a device-resident id, with the expert weight applied in the epilogue."""
    nE, k, E, F = 8, 2, 512, 768
    g = torch.Generator().manual_seed(31)
    logits = torch.randn(3, nE, generator=g).to(DEV)
    ids, w = ops.moe_route(logits, k)
    pr = torch.softmax(logits, -1)
    tw, ti = pr.topk(k, -1)
    assert torch.equal(ids.view(3, k).long(), ti)
    assert torch.allclose(w.view(3, k), tw / tw.sum(-1, keepdim=True), atol=1e-6)
    # stacked experts
    gate = torch.randn(nE * F, E, generator=g) * 0.05
    up = torch.randn(nE * F, E, generator=g) * 0.05
    down = torch.randn(nE * E, F, generator=g) * 0.05
    Wg, Wu, Wd = (DeviceWeight.from_dense(m, t, DEV) for m in (gate, up, down))
    from distributed_llm_pipeline_b200.gguf.quants import dequantize, quantize
    import numpy as np
    deq = lambda m: torch.from_numpy(dequantize(quantize(m.numpy(), t), t, tuple(m.shape)).astype(np.float32)).to(DEV)
    dg, du, dd = deq(gate), deq(up), deq(down)
    h = torch.randn(1, E, generator=g).to(DEV)
    nw = (torch.rand(E, generator=g) + 0.5).to(DEV)
    xn = (h * torch.rsqrt(h.pow(2).mean(-1, keepdim=True) + 1e-5) * nw).half().float()
    href = h.clone()
    hout = h.clone()
    act = torch.empty(k, F, dtype=torch.float16, device=DEV)
    for j in range(k):
        e = int(ids[j])
        ops.gemv_moe(Wg, h, act[j:j + 1], "swiglu", ids[j:j + 1], F, w_up=Wu, norm_w=nw, eps=1e-5)
        a_ref = torch.nn.functional.silu(xn @ dg[e * F:(e + 1) * F].T) * (xn @ du[e * F:(e + 1) * F].T)
        assert nmse(a_ref, act[j:j + 1]) < (3e-4 if t.name.startswith("Q") else 2e-5)
        href += float(w[j]) * (act[j:j + 1].float() @ dd[e * E:(e + 1) * E].T)
    for j in range(k):
        ops.gemv_moe(Wd, act[j:j + 1], hout, "add", ids[j:j + 1], E, out_scale=w[j:j + 1])
    assert nmse(href, hout) < (1e-4 if t.name.startswith("Q") else 1e-6)


@pytest.mark.parametrize("t", [GGMLType.F16, GGMLType.Q8_0, GGMLType.Q4_K])
@pytest.mark.parametrize("T,nE,k", [(1, 4, 2), (7, 8, 2), (64, 8, 2), (300, 8, 2), (33, 60, 4), (129, 128, 8)])
def test_moe_grouped_gemm_pipeline(t, T, nE, k):
    """route -> plan -> gather -> grouped SwiGLU GEMM -> grouped down GEMM -> combine, against per-token fp32 math with the
    same (dequantised) expert weights.  Covers experts that receive no token, partial token tiles and > 32 experts."""
    from distributed_llm_pipeline_b200.gguf.quants import dequantize, quantize
    import numpy as np
    E, F = 256, 256
    g = torch.Generator().manual_seed(100 + T + nE)
    logits = torch.randn(T, nE, generator=g).to(DEV)
    if T >= 64:
        logits[:, 1] = -30.0                                   # expert 1 never selected: an empty group in the plan
    A = T * k
    ids = torch.zeros(A, dtype=torch.int32, device=DEV)
    w = torch.zeros(A, dtype=torch.float32, device=DEV)
    for renorm in (True, False):
        ops.moe_route_ex(logits, nE, k, renorm, ids, w)
        pr = torch.softmax(logits, -1)
        tw, ti = pr.topk(k, -1)
        assert torch.equal(ids.view(T, k).long(), ti)
        assert torch.allclose(w.view(T, k), tw / tw.sum(-1, keepdim=True) if renorm else tw, atol=1e-6)
    bt = 16 if A // nE <= 16 else 32 if A // nE <= 32 else 64
    plan = ops.MoePlan(A, nE, DEV)
    ops.moe_plan(ids, nE, bt, plan)
    pos, src, bounds = plan.pos.long(), plan.src.long(), plan.bounds.tolist()
    assert bounds[0] == 0 and bounds[-1] == A
    assert torch.equal(src[pos], torch.arange(A, device=DEV))                     # a permutation ...
    for e in range(nE):
        rows = src[bounds[e]:bounds[e + 1]]
        assert bool((ids[rows] == e).all()) and bool((rows[1:] > rows[:-1]).all())   # ... grouped by expert, stable in token order
    nt = int(plan.n_tiles)
    assert nt == sum((bounds[e + 1] - bounds[e] + bt - 1) // bt for e in range(nE))
    assert int(plan.tile_rows[:nt].sum()) == A
    gate = torch.randn(nE * F, E, generator=g) * 0.05
    up = torch.randn(nE * F, E, generator=g) * 0.05
    down = torch.randn(nE * E, F, generator=g) * 0.05
    Wg, Wu, Wd = (DeviceWeight.from_dense(m, t, DEV) for m in (gate, up, down))
    deq = lambda m: torch.from_numpy(dequantize(quantize(m.numpy(), t), t, tuple(m.shape)).astype(np.float32)).to(DEV)
    dg, du, dd = deq(gate), deq(up), deq(down)
    x = torch.randn(T, E, generator=g).half().to(DEV)
    xs = torch.zeros(A, E, dtype=torch.float16, device=DEV)
    ops.moe_gather(x, plan, k, A, xs)
    assert torch.equal(xs, x[src // k])
    act = torch.zeros(A, F, dtype=torch.float16, device=DEV)
    ops.linear_grouped(Wg, xs, act, "swiglu", nE, F, bt, plan, w_up=Wu)
    y = torch.zeros(A, E, dtype=torch.float32, device=DEV)
    ops.linear_grouped(Wd, act, y, "f32", nE, E, bt, plan)
    h = torch.randn(T, E, generator=g).to(DEV)
    h_ref = h.clone()
    ops.moe_combine(y, plan, w, T, k, h)
    tol = 3e-4 if t.name.startswith("Q") else 2e-5
    for e in range(nE):
        sel = (ids == e).nonzero().flatten()
        if sel.numel() == 0:
            continue
        xe = x[sel // k].float()
        a_ref = torch.nn.functional.silu(xe @ dg[e * F:(e + 1) * F].T) * (xe @ du[e * F:(e + 1) * F].T)
        assert nmse(a_ref, act[pos[sel]]) < tol, e
        y_ref = act[pos[sel]].float() @ dd[e * E:(e + 1) * E].T
        assert nmse(y_ref, y[pos[sel]]) < tol, e
        h_ref.index_add_(0, sel // k, w[sel][:, None] * y[pos[sel]])
    assert nmse(h_ref, h) < 1e-6


@pytest.mark.parametrize("t", [GGMLType.F16, GGMLType.Q8_0, GGMLType.Q4_K])
@pytest.mark.parametrize("T", [5, 8, 32, 64, 200])
@pytest.mark.parametrize("mode", ["f16", "f32", "add", "swiglu"])
def test_gemm_split_k_workspace_fixup(t, T, mode):
    """Skinny problems (few 128-row tiles) split K across CTAs through the workspace; the last split adds the partials in split
    order, so the result matches the fp32 reference and is bit-identical from run to run and to the unsplit kernel's rounding
    class.  N = 384 gives 3 tiles -> 8 splits of K = 4096."""
    from distributed_llm_pipeline_b200.gguf.quants import dequantize, quantize
    import numpy as np
    N, K = 384, 4096
    g = torch.Generator().manual_seed(7 + T)
    w = torch.randn(N, K, generator=g) * 0.03
    w2 = torch.randn(N, K, generator=g) * 0.03
    x = torch.randn(T, K, generator=g).half().to(DEV)
    W, W2 = DeviceWeight.from_dense(w, t, DEV), DeviceWeight.from_dense(w2, t, DEV)
    deq = lambda m: torch.from_numpy(dequantize(quantize(m.numpy(), t), t, tuple(m.shape)).astype(np.float32)).to(DEV)
    y_ref = x.float() @ deq(w).T
    if mode == "swiglu":
        y_ref = torch.nn.functional.silu(y_ref) * (x.float() @ deq(w2).T)
    outs = []
    for rep in range(2):
        if mode == "add":
            out = torch.ones(T, N, device=DEV)
            ops.linear(W, x, "add", out=out)
            got = out - 1.0
        else:
            got = ops.linear(W, x, mode, w_up=W2 if mode == "swiglu" else None).float()
        outs.append(got.clone())
    tol = 4e-4 if t.name.startswith("Q") else (1e-5 if mode in ("f32", "add") else 2e-5)
    assert nmse(y_ref, outs[0]) < tol
    if mode != "add":          # (the residual-add epilogue reduces its splits with atomics: order, hence rounding, may differ)
        assert torch.equal(outs[0], outs[1])
    ws = ops.gemm_workspace(torch.device(DEV))
    assert int(ws[:16384].view(torch.int32).abs().sum()) == 0          # every tile counter went back to zero


def test_rope_rows_of_a_prompt():
    """RoPE of many tokens at once (one block a token) against the one-pair-a-thread kernel: whole and partial rotation, both pairings, negative slots."""
    T, Hq, Hkv, page = 130, 80, 8, 16             # (fewer heads: the other kernel as well)
    for D, n_rot in ((64, 64), (128, 128), (128, 96), (64, 32)):
        for neox in (False, True):
            g = torch.Generator(DEV).manual_seed(D + n_rot)
            qkv = torch.randn(T, (Hq + 2 * Hkv) * D, device=DEV, generator=g).half()
            pos = torch.randint(0, 5000, (T,), device=DEV, generator=g).to(torch.int32)
            slot = torch.randperm(T + 40, device=DEV, generator=g)[:T].to(torch.int32)
            slot[::7] = -1
            inv = (10000.0 ** (-torch.arange(0, n_rot // 2).double() * 2 / n_rot)).float().to(DEV)
            got, want = ([torch.zeros(T, Hq * D, device=DEV, dtype=torch.float16)] + [torch.zeros(12, Hkv, page, D, device=DEV, dtype=torch.float16) for _ in range(2)] for _ in range(2))
            ops.rope_kv(qkv, pos, slot, inv, got[1], got[2], Hq, Hkv, D, neox, q_out=got[0])
            for i in range(0, T, 5):                    # (few tokens: the other kernel)
                ops.rope_kv(qkv[i:i + 5], pos[i:i + 5], slot[i:i + 5], inv, want[1], want[2], Hq, Hkv, D, neox, q_out=want[0][i:i + 5])
            for a, b in zip(got, want):
                assert nmse(b, a) < 1e-8, (D, n_rot, neox)


def test_a_wait_that_runs_out_is_an_error_once(tmp_models):
    """A wait that nothing ends returns after its limit and raises the status: the engine's next call fails, the one after it works, and the kernels wait again.  The
    status is also there for callers that ask for it with a synchronisation."""
    from distributed_llm_pipeline_b200.models.llama import LlamaEngine
    from distributed_llm_pipeline_b200.models.weights import load_weights
    from distributed_llm_pipeline_b200.ops import layers as lops
    from distributed_llm_pipeline_b200.ops import lib as L
    lib, flag = L.load(), ctypes.c_int(0)
    eng = LlamaEngine(load_weights(tmp_models[("tiny", "F16")], "cuda"), n_ctx=256, max_seqs=1, page_size=16, max_batch_tokens=64)
    L.check_waits()
    L.check(lib.dlp_set_wait_limit(0.02), "set_wait_limit")
    try:
        sid = eng.alloc_seq()
        want = eng.prefill(sid, list(range(1, 20))).clone()
        for again in (lambda: eng.prefill(sid, [5]), lambda: eng.decode([sid], [5], sample=False)):
            L.check(lib.dlp_wait_probe(None), "wait_probe")
            torch.cuda.synchronize()
            L.check(lib.dlp_gemm_wait_expired(ctypes.byref(flag)), "wait_expired")
            assert flag.value == 1
            with pytest.raises(L.WaitError):
                again()
            L.check(lib.dlp_gemm_wait_expired(ctypes.byref(flag)), "wait_expired")
            assert flag.value == 0
            eng.truncate_seq(sid, 0)
            assert torch.equal(eng.prefill(sid, list(range(1, 20))), want)
            again()
        L.check(lib.dlp_wait_probe(None), "wait_probe")
        with pytest.raises(L.WaitError):
            lops.check_waits()
        lops.check_waits()
    finally:
        L.check(lib.dlp_set_wait_limit(2.0), "set_wait_limit")
    assert lib.dlp_set_wait_limit(0.0) != 0


@pytest.mark.parametrize("t,bt", [(GGMLType.F16, 64), (GGMLType.F16, 128), (GGMLType.BF16, 128), (GGMLType.Q4_K, 64), (GGMLType.Q8_0, 64), (GGMLType.Q6_K, 64), (GGMLType.Q5_K, 64)])
@pytest.mark.parametrize("rows", [[700, 1, 0, 129], [64, 63, 65, 300]])
def test_grouped_products_of_long_prompts(t, bt, rows):
    """Experts with several tiles of tokens (dense weights on pairs of SMs, block types in tiles of 64), with one token and with none, against 64 bits."""
    nE, E, F, A = len(rows), 768, 512, sum(rows)
    half = torch.bfloat16 if t == GGMLType.BF16 else torch.float16
    ids = torch.repeat_interleave(torch.arange(nE), torch.tensor(rows)).to(torch.int32).to(DEV)
    plan = ops.MoePlan(A, nE, DEV)
    ops.moe_plan(ids, nE, bt, plan)
    assert int(plan.n_tiles) == sum((n + bt - 1) // bt for n in rows)
    (Wg, dg), (Wu, du), (Wd, dd) = _w(nE * F, E, t, 1), _w(nE * F, E, t, 2), _w(nE * E, F, t, 3)
    x = torch.randn(A, E, device=DEV, generator=torch.Generator(DEV).manual_seed(5)).to(half)
    z = torch.randn(A, F, device=DEV, generator=torch.Generator(DEV).manual_seed(6)).to(half)
    act, y = torch.zeros(A, F, dtype=torch.float16, device=DEV), torch.zeros(A, E, device=DEV)
    if t != GGMLType.BF16:            # (the gated epilogue of bf16 weights is bf16)
        ops.linear_grouped(Wg, x, act, "swiglu", nE, F, bt, plan, w_up=Wu)
    ops.linear_grouped(Wd, z, y, "f32", nE, E, bt, plan)
    at = 0
    for e, n in enumerate(rows):
        if n:
            xe, ze = x[at:at + n].double(), z[at:at + n].double()
            g, u, d = (m[e * r:(e + 1) * r].double() for m, r in ((dg, F), (du, F), (dd, E)))
            assert nmse(ze @ d.T, y[at:at + n]) < 2e-7, e
            if t != GGMLType.BF16:
                assert nmse(torch.nn.functional.silu(xe @ g.T) * (xe @ u.T), act[at:at + n]) < 2e-6, e
        at += n
