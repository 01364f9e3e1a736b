"""Parity of every CUDA kernel with a CPU statement of the same op, called through the
C ABI (ctypes on raw device pointers), on seeded inputs.  Integer/byte work must be
bit-exact; floating point uses the op-level tolerance of the reference's CUDA tests
(rtol 5e-2 / atol 1e-2, tests/test_cuda_executor.py:150-319), tightened where bf16 allows."""

import ctypes as C
import math
import subprocess

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

DT = {torch.float32: 0, torch.float16: 1, torch.bfloat16: 2, torch.int32: 3, torch.int64: 4, torch.uint8: 5}


@pytest.fixture(scope="module")
def lib(native_lib):
    assert torch.cuda.is_available()
    torch.cuda.set_device(0)
    return native_lib


def ok(lib, rc):
    assert rc == 0, lib.b200_last_error().decode()
    torch.cuda.synchronize()


def go(lib, rc):
    """The call was taken; nothing waits for it (the next launch may follow at once)."""
    assert rc == 0, lib.b200_last_error().decode()


def stream():
    return torch.cuda.current_stream().cuda_stream


def gen(shape, dtype=torch.bfloat16, seed=0, scale=1.0):
    return (torch.randn(*shape, generator=torch.Generator().manual_seed(seed)) * scale).to(dtype)


def bt(t):
    from cuda_runtime import native

    return native.make_tensor(t.data_ptr(), str(t.dtype).replace("torch.", ""), tuple(t.shape), tuple(t.stride()))


class _KernelNode(C.Structure):   # CUDA_KERNEL_NODE_PARAMS of the driver API, version 2
    _fields_ = [("func", C.c_void_p), ("dims", C.c_uint * 7), ("params", C.c_void_p), ("extra", C.c_void_p), ("kern", C.c_void_p), ("ctx", C.c_void_p)]


def kernels_of(call):
    """Names of the kernels that a call launches: the nodes of a graph that it is captured into.  (The profiler now and then
    reports nothing, more often the more tests ran before.)"""
    call()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        call()
    cu = C.CDLL("libcuda.so.1")
    raw, n, names = C.c_void_p(graph.raw_cuda_graph()), C.c_size_t(0), []
    assert cu.cuGraphGetNodes(raw, None, C.byref(n)) == 0
    nodes = (C.c_void_p * n.value)()
    assert cu.cuGraphGetNodes(raw, nodes, C.byref(n)) == 0
    for node in nodes:
        kind, p, name = C.c_int(-1), _KernelNode(), C.c_char_p()
        assert cu.cuGraphNodeGetType(C.c_void_p(node), C.byref(kind)) == 0
        if kind.value != 0:   # not a kernel
            continue
        assert cu.cuGraphKernelNodeGetParams_v2(C.c_void_p(node), C.byref(p)) == 0
        assert (cu.cuFuncGetName(C.byref(name), C.c_void_p(p.func)) if p.func else cu.cuKernelGetName(C.byref(name), C.c_void_p(p.kern))) == 0
        names.append(subprocess.run(["c++filt", name.value.decode()], capture_output=True, text=True, check=True).stdout)
    return names


def close(got, ref, rtol=2e-2, atol=1e-2):
    np.testing.assert_allclose(got.float().cpu().numpy(), ref.float().cpu().numpy(), rtol=rtol, atol=atol)


# ------------------------------------------------------------------ linear
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("M,N,K,bias,res,relu,silu", [
    (777, 2048, 1536, True, False, False, False),   # one wave of 128-wide tiles, ragged last row tile
    (777, 1536, 1536, False, True, False, False),   # the same with a residual
    (1537, 716, 1032, True, True, True, False),     # the same with ragged columns, rows and k: rows that are no whole 16-byte words
    (1537, 720, 1032, True, True, True, False),     # ragged columns in whole words: bulk copies
    (777, 1536, 3080, False, True, False, False),   # a reduction past the bulk copies' limit
    (777, 1500, 3080, True, True, False, False),
    (1537, 700, 1032, True, True, True, False),     # 143 64-wide tiles: one wave of them
    (900, 1400, 1096, True, False, False, True),
    (1, 1536, 1536, True, False, False, False),
    (1, 1536, 8960, False, True, False, False),
    (8, 8960, 1536, False, False, False, True),
    (64, 256, 1536, True, False, False, False),
    (3, 1000, 512, True, False, True, False),
    (7, 130, 72, True, True, True, False),
    (65, 1536, 1536, True, True, False, False),
    (512, 8960, 1536, False, False, False, True),
    (300, 1000, 2048, True, False, True, False),
    (128, 151936 // 8, 1536, False, False, False, False),
    # 256 x 256 tiles on CTA pairs: row tail (640 = 2 * 256 + 128), column tail, K tail, every epilogue term
    (640, 8200, 1088, True, True, True, False),
    (300, 16384, 1024, True, False, False, False),
    (512, 8960, 1536, True, True, False, True),
    # few 256 x 256 tiles, long reduction: the pairs split K, a second kernel adds the fp32 partial sums
    (1024, 1536, 8960, True, True, False, False),
    (512, 1536, 8960, False, True, False, False),
    (1000, 1200, 4104, False, False, True, False),
])
def test_linear(lib, dtype, M, N, K, bias, res, relu, silu):
    a, w = gen((M, K), dtype), gen((N, K), dtype, 1, 0.05)
    b = gen((N,), dtype, 2) if bias else None
    r = gen((M, N), dtype, 3) if res else None
    u = gen((M, N), dtype, 4) if silu else None
    ref = a.float() @ w.float().t()
    if bias:
        ref = ref + b.float()
    if res:
        ref = ref.to(dtype).float() + r.float()
    if relu:
        ref = torch.relu(ref)
    if silu:
        s = ref.to(dtype).float()
        ref = torch.nn.functional.silu(s).to(dtype).float() * u.float()
    A, W = a.cuda(), w.cuda()
    Bv, Rv, Uv = (t.cuda() if t is not None else None for t in (b, r, u))
    out = torch.full((M, N), float("nan"), dtype=dtype, device="cuda")
    nbytes = lib.b200_linear_workspace_bytes(M, N, K)
    ws = torch.zeros(max(nbytes, 16), dtype=torch.uint8, device="cuda")
    p = lambda t: t.data_ptr() if t is not None else None
    for _ in range(2):  # second call checks that the split-K workspace was left clean
        out.fill_(float("nan"))
        ok(lib, lib.b200_linear(p(A), p(W), p(Bv), p(Rv), p(out), M, N, K, K, K, N, N, DT[dtype], DT[dtype],
                                (1 if relu else 0) | (2 if silu else 0), p(Uv), N, p(ws), ws.numel(), stream()))
        close(out, ref, rtol=2e-2, atol=2e-2 * max(1.0, math.sqrt(K) * 0.05))
    assert not ws.any()
    code = C.c_int(-1)
    ok(lib, lib.b200_debug_device_error(C.byref(code), 1))
    assert code.value == 0, f"a bounded wait in the tcgen05 GEMM gave up (code {code.value})"


@pytest.mark.parametrize("M,N,K", [(128, 128, 64), (129, 200, 72), (1000, 1536, 1536), (512, 151936, 1536)])
def test_linear_tcgen05_shapes(lib, M, N, K):
    """Large-M linears take the tcgen05/TMEM path: tile edges, K tails and a very wide N."""
    dtype = torch.bfloat16
    a, w = gen((M, K), dtype), gen((N, K), dtype, 1, 0.05)
    A, W = a.cuda(), w.cuda()
    out = torch.full((M, N), float("nan"), dtype=dtype, device="cuda")
    ok(lib, lib.b200_linear(A.data_ptr(), W.data_ptr(), None, None, out.data_ptr(), M, N, K, K, K, N, 0, 2, 2, 0, None, 0, None, 0, stream()))
    ref = (A.float() @ W.float().t())           # fp32 GEMM on the device as the large-size reference
    err = (out.float() - ref).abs().max().item()
    assert err <= 2e-2 * max(1.0, math.sqrt(K) * 0.05) + 1e-2 * ref.abs().max().item(), err
    if N <= 2048:
        close(out, a.float() @ w.float().t(), rtol=2e-2, atol=2e-2 * max(1.0, math.sqrt(K) * 0.05))
    code = C.c_int(-1)
    ok(lib, lib.b200_debug_device_error(C.byref(code), 1))
    assert code.value == 0


@pytest.mark.parametrize("M,I,K", [(1, 8960, 1536), (8, 8960, 1536), (64, 8960, 1536), (512, 8960, 1536), (40, 256, 72)])
def test_linear_gated_mlp_epilogue(lib, M, I, K):
    """silu(x Wg^T) * (x Wu^T) from one GEMM over gate/up rows interleaved in blocks of 64."""
    dtype = torch.bfloat16
    x, wg, wu = gen((M, K), dtype), gen((I, K), dtype, 1, 0.05), gen((I, K), dtype, 2, 0.05)
    g = (x.float() @ wg.float().t()).to(dtype).float()
    u = (x.float() @ wu.float().t()).to(dtype).float()
    ref = torch.nn.functional.silu(g).to(dtype).float() * u
    merged = torch.stack([wg.view(I // 64, 64, K), wu.view(I // 64, 64, K)], 1).reshape(2 * I, K).contiguous()
    X, W = x.cuda(), merged.cuda()
    out = torch.full((M, I), float("nan"), dtype=dtype, device="cuda")
    ws = torch.zeros(max(lib.b200_linear_workspace_bytes(M, 2 * I, K), 16), dtype=torch.uint8, device="cuda")
    for _ in range(2):
        ok(lib, lib.b200_linear(X.data_ptr(), W.data_ptr(), None, None, out.data_ptr(), M, 2 * I, K, K, K, I, 0, 2, 2, 4, None, 0,
                                ws.data_ptr(), ws.numel(), stream()))
        close(out, ref, rtol=3e-2, atol=3e-2 * max(1.0, math.sqrt(K) * 0.05))
    assert not ws.any()


@pytest.mark.parametrize("M,N,K,mode", [(1, 2048, 1536, "bias"), (8, 2048, 1536, "bias"), (64, 2048, 1536, "bias"), (64, 17920, 1536, "glu"),
                                        (5, 17920, 1536, "glu"), (64, 151936, 1536, "plain"), (33, 1536, 1536, "chain"), (64, 1536, 8960, "chain"),
                                        *((m, 1536, 1536, "chain") for m in (1, 8, 9, 16, 17, 24, 25)),
                                        *((m, 1536, 8960, "chain") for m in (1, 9, 16, 17)), *((m, 17920, 1536, "glu") for m in (8, 9, 16, 17)),
                                        *((m, 2048, 1536, "bias") for m in (9, 17, 24)), (24, 4096, 1536, "glu")])
def test_linear_norm_fused_rmsnorm(lib, M, N, K, mode):
    """RMSNorm folded into decode GEMMs.  "chain": a residual GEMM that also writes the sum-of-squares
    partials of its output rows, followed by a GEMM over gain-folded weights that scales its output
    rows by 1/rms from those partials - against the fp32 statement of rmsnorm + matmul with the
    roundings of the unfused kernels, and against the unfused kernels themselves."""
    dtype = torch.bfloat16
    BF = 2
    if mode == "chain":
        a, w, res = gen((M, K), dtype, 0, 0.5), gen((N, K), dtype, 1, 0.05), gen((M, N), dtype, 2)
        y = torch.empty(M, N, dtype=dtype, device="cuda")
        sq = torch.full((M, N // 64), float("nan"), device="cuda")
        A, W, R = a.cuda(), w.cuda(), res.cuda()
        ok(lib, lib.b200_linear_norm(A.data_ptr(), W.data_ptr(), None, R.data_ptr(), y.data_ptr(), M, N, K, K, K, N, N, BF, BF, 8,
                                     0.0, None, 0, sq.data_ptr(), stream()))
        ref = ((a.float() @ w.float().T).to(dtype).float() + res.float()).to(dtype)
        close(y, ref, rtol=2e-2, atol=2e-2)
        # the partials describe the rows that were actually written
        want_sq = y.float().pow(2).reshape(M, N // 64, 64).sum(-1)
        torch.testing.assert_close(sq, want_sq, rtol=1e-4, atol=1e-4)
        x, n_part, sumsq = y, N // 64, sq       # feed the next layer from them
        K2, N2 = N, 2048
    else:
        x = gen((M, K), dtype, 0, 3.0).cuda()
        n_part = 3
        sumsq = x.float().pow(2).reshape(M, n_part, K // n_part).sum(-1).contiguous()
        K2, N2 = K, N
    gain = (1 + 0.1 * gen((K2,), torch.float32, 5)).to(dtype).cuda()
    w2 = gen((N2, K2), dtype, 6, 0.03).cuda()
    w2_folded = (w2.float() * gain.float()[None, :]).to(dtype)          # what the weight preparation produces
    bias = gen((N2,), dtype, 7).cuda() if mode in ("bias", "chain") else None
    epi = 8 | (4 if mode == "glu" else 0)
    n_out = N2 // 2 if mode == "glu" else N2
    out = torch.full((M, n_out), float("nan"), dtype=dtype, device="cuda")
    ok(lib, lib.b200_linear_norm(x.data_ptr(), w2_folded.data_ptr(), bias.data_ptr() if bias is not None else None, None, out.data_ptr(), M, N2, K2,
                                 K2, K2, n_out, 0, BF, BF, epi, 1e-6, sumsq.data_ptr(), n_part, None, stream()))

    def finish(r):
        if bias is not None:
            r = r + bias.float().cpu()
        if mode == "glu":
            r = r.reshape(M, N2 // 128, 2, 64)
            g_, u_ = r[:, :, 0].to(dtype).float(), r[:, :, 1].to(dtype).float()
            r = (torch.nn.functional.silu(g_).to(dtype).float() * u_).reshape(M, n_out)
        return r

    xf = x.float().cpu()
    rr = torch.rsqrt(xf.pow(2).mean(-1, keepdim=True) + 1e-6)
    # the reference's rounding points: round(x r), round(. * gain), then the GEMM
    a2 = ((xf * rr).to(dtype).float() * gain.float().cpu()).to(dtype).float()
    # (the gated form multiplies two rounded factors: a one-ulp difference in the gate is scaled by |up| <= ~5)
    tol = 6e-2 if mode == "glu" else 3e-2
    close(out, finish(a2 @ w2.float().cpu().T), rtol=3e-2, atol=tol)
    # the exact statement of what the kernel computes: r * (x W'^T)
    close(out, finish(rr * (xf @ w2_folded.float().cpu().T)), rtol=2e-2, atol=tol / 2)
    # and the unfused pair of kernels
    y_n = torch.empty_like(x)
    ok(lib, lib.b200_rmsnorm(x.data_ptr(), gain.data_ptr(), y_n.data_ptr(), M, K2, K2, K2, 1e-6, BF, 1, stream()))
    out2 = torch.empty_like(out)
    ok(lib, lib.b200_linear(y_n.data_ptr(), w2.data_ptr(), bias.data_ptr() if bias is not None else None, None, out2.data_ptr(), M, N2, K2,
                            K2, K2, n_out, 0, BF, BF, epi, None, 0, None, 0, stream()))
    close(out, out2, rtol=3e-2, atol=tol)
    code = C.c_int(0)
    ok(lib, lib.b200_debug_device_error(C.byref(code), 1))
    assert code.value == 0


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("M", [1, 8, 9, 16, 17, 24, 25])
@pytest.mark.parametrize("N,K,shift,ldx", [
    (64, 64, 0, 0),           # one block, one chunk: three of the four warps have none
    (128, 320, 0, 16),        # five chunks, strided rows
    (192, 2112, 16, 0),       # eight splits of uneven length; W 32-byte aligned inside its buffer
    (192, 2112, 8, 0),        # W only 16-byte aligned: the tensor-map kernel
    (64 * 300, 192, 0, 0),    # more blocks than resident CTAs: a CTA walks two
    (64 * 150, 25664, 0, 0),  # no split and rows too long to keep: the tensor-map kernel
    (64 * 150, 1536, 0, 0),   # no split: two groups of rows fit beside a second CTA, three do not
    (64 * 148, 1024, 0, 0),   # one block per SM: two splits
    (64 * 97, 1088, 0, 0),    # two splits, 9 and 8 chunks
    (64 * 112, 960, 0, 0),    # one block per SM, all chunks in flight at once: no split
    (64 * 56, 1792, 0, 0),    # four splits of seven chunks
    (64 * 56, 1536, 0, 0),    # three splits of eight
    (200, 328, 0, 0),         # ragged block and chunk
])
def test_linear_few_rows_edges(lib, M, N, K, shift, ldx, dtype):
    """Edges of the weight-streaming kernel and of its rule; residual, bias and ReLU in the final pass.  The bound: fp32
    sums in any order (K * 2^-24 of the sum of magnitudes, products exact), and two roundings to
    the activation type (8 or 11 significant bits: at most 2^-8 or 2^-11 of the value each; subnormal halves 2^-25)."""
    lda, ldo = K + ldx, N + ldx
    A = torch.full((M, lda), float("nan"), dtype=dtype, device="cuda")
    A[:, :K] = gen((M, K), dtype).cuda()
    g = torch.Generator(device="cuda").manual_seed(1)
    Wb = torch.randn(N * K + shift, generator=g, device="cuda").mul_(K ** -0.5).to(dtype)
    W = Wb[shift:].view(N, K)
    b, r = gen((N,), dtype, seed=2).cuda(), torch.zeros(M, ldo, dtype=dtype, device="cuda")
    r[:, :N] = gen((M, N), dtype, seed=3).cuda()
    out = torch.full((M, ldo), 7.0, dtype=dtype, device="cuda")
    ws = torch.zeros(1 << 22, dtype=torch.uint8, device="cuda")
    ok(lib, lib.b200_linear(A.data_ptr(), W.data_ptr(), b.data_ptr(), r.data_ptr(), out.data_ptr(), M, N, K, lda, K, ldo, ldo, DT[dtype], DT[dtype],
                            1 | 8, None, 0, ws.data_ptr(), ws.numel(), stream()))
    x, w = A[:, :K].double(), W.double()
    lin = x @ w.T + b.double()
    want = (lin + r[:, :N].double()).clamp(min=0)
    bound = (x.abs() @ w.abs().T) * (K * 2.0 ** -24) + (lin.abs() + want) * (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11) * 1.01 + 1e-6
    err = (out[:, :N].double() - want).abs()
    assert (err <= bound).all(), float((err - bound).max())
    assert (out[:, N:] == 7.0).all()


@pytest.mark.parametrize("M,N,K,res,kernel", [
    (1, 1536, 8960, True, "gemm_stream_kernel"), (16, 1536, 8960, True, "gemm_stream_kernel"), (17, 1536, 8960, True, "gemm_tc5_kernel"),
    (24, 2048, 1536, False, "gemm_stream_kernel"), (25, 2048, 1536, False, "gemm_tc5_kernel"),
    (16, 17920, 1536, False, "gemm_stream_kernel"), (17, 17920, 1536, False, "gemm_tc5_kernel"), (8, 200, 328, False, "gemm_tc5_kernel"),
    (777, 2048, 1536, False, "gemm_tc5_kernel"), (777, 1536, 1536, True, "gemm_tc5p_kernel"), (777, 1500, 1536, True, "gemm_tc5_kernel"),
    (2048, 1536, 1536, True, "gemm_pair_kernel"),
    (65, 9472, 1536, False, "gemm_tc5_kernel"), (128, 9472, 1536, False, "gemm_tc5_kernel"), (129, 9472, 1536, False, "gemm_pair_kernel"),
    (65, 9480, 1536, False, "gemm_pair_kernel"), (128, 17920, 1536, False, "gemm_pair_kernel"), (64, 17920, 1536, False, "gemm_tc5_kernel"),
])
def test_linear_runs_on_the_kernel_that_its_shape_calls_for(lib, M, N, K, res, kernel):
    t = torch.zeros(M * K + N * K + 2 * M * N, dtype=torch.bfloat16, device="cuda")
    a, w, o, r = (t[n:].data_ptr() for n in (0, M * K, M * K + N * K, M * K + N * K + M * N))
    ran = kernels_of(lambda: go(lib, lib.b200_linear(a, w, None, r if res else None, o, M, N, K, K, K, N, N if res else 0, 2, 2, 8, None, 0, None, 0, stream())))
    assert len(ran) == 1 and kernel + "<" in ran[0], ran


@pytest.mark.parametrize("M", [1, 9, 24, 25, 64])
def test_row_scale_adds_its_partials_in_index_order(lib, M):
    """Every kernel behind b200_linear_norm adds the sum-of-squares partials of a row in index order: 2^24 and then ones
    is 2^24 that way, and up to 2^24 + 24 in any other (two sums of eight ones and more survive the rounding).  An fp32
    bias takes the product with the right factor away again, so what is left is the factor's error: a few roundings of
    2^-24 against 2^-20.4 for the other order."""
    N, K, parts = 2048, 1536, 32
    ss = torch.ones(M, parts)
    ss[:, 0] = 2.0 ** 24
    ss *= (4.0 ** (torch.arange(M) % 3))[:, None]
    total = ss[:, 0]                                   # the ones vanish one by one
    for j in range(1, parts):
        assert (total + ss[:, j] == total).all()
    x = torch.zeros(M, K)
    x[:, 0] = total.div(K).sqrt().bfloat16().float()   # one product per output: its sum is exact in any order
    w = torch.zeros(N, K)
    w[:, 0] = gen((N,), seed=3).float()
    prod = x[:1, 0] * w[:, 0]                          # the bias is shared by the rows, so they all get the first row's product
    x[:, 0] = x[0, 0] * 2.0 ** (torch.arange(M) % 3)
    rinv = 1.0 / torch.sqrt(total / K + 1e-6)
    bias = -(prod * rinv[0])
    X, W, B, SQ = x.bfloat16().cuda(), w.bfloat16().cuda(), bias.cuda(), ss.cuda()
    out = torch.full((M, N), float("nan"), dtype=torch.bfloat16, device="cuda")
    ok(lib, lib.b200_linear_norm(X.data_ptr(), W.data_ptr(), B.data_ptr(), None, out.data_ptr(), M, N, K, K, K, N, 0, 2, 0, 8, 1e-6,
                                 SQ.data_ptr(), parts, None, stream()))
    assert (out.float().cpu().abs() <= prod.mul(rinv[0]).abs() * 2.0 ** -22).all()


def test_linear_norm_rejects_shapes_outside_the_fused_kernel(lib):
    t = torch.zeros(128 * 1536, dtype=torch.bfloat16, device="cuda")
    f = torch.zeros(4096, device="cuda")
    args = lambda M, N, K, cols, sq_out: (t.data_ptr(), t.data_ptr(), None, None, t.data_ptr(), M, N, K, K, K, N, 0, 2, 2, 0, 1e-6,
                                          f.data_ptr(), cols, f.data_ptr() if sq_out else None, stream())
    assert lib.b200_linear_norm(*args(100, 64, 128, 1, False)) == -4 and b"M <= 64" in lib.b200_last_error()   # prefill-sized M
    assert lib.b200_linear_norm(*args(8, 64, 128, 40, False)) == -4                                              # too many partials
    assert lib.b200_linear_norm(*args(8, 72, 128, 1, True)) == -4                                                # N not a multiple of 64


def test_bounded_wait_runs_out_and_the_context_survives(lib):
    """A barrier wait that can never be satisfied: the kernel's bounded wait gives up after the probe limit,
    leaves code 99 in the device error word and returns; the next kernels run normally."""
    code = C.c_int(-1)
    ok(lib, lib.b200_debug_device_error(C.byref(code), 1))
    assert code.value == 0
    ok(lib, lib.b200_debug_wait_timeout(2000, stream()))
    ok(lib, lib.b200_debug_device_error(C.byref(code), 0))
    assert code.value == 99
    ok(lib, lib.b200_debug_device_error(C.byref(code), 1))     # reads 99 again and clears
    ok(lib, lib.b200_debug_device_error(C.byref(code), 0))
    assert code.value == 0
    a, w = gen((4, 256)), gen((128, 256), seed=1)
    out = torch.empty(4, 128, dtype=torch.bfloat16, device="cuda")
    A, W = a.cuda(), w.cuda()
    ok(lib, lib.b200_linear(A.data_ptr(), W.data_ptr(), None, None, out.data_ptr(), 4, 128, 256, 256, 256, 128, 0, 2, 2, 0, None, 0, None, 0, stream()))
    close(out, a.float() @ w.float().T, rtol=2e-2, atol=2e-2)
    assert lib.b200_debug_wait_timeout(0, stream()) == -1


def test_linear_rejects_unaligned(lib):
    a = torch.zeros(4, 12, dtype=torch.bfloat16, device="cuda")
    rc = lib.b200_linear(a.data_ptr(), a.data_ptr(), None, None, a.data_ptr(), 4, 4, 12, 12, 12, 4, 0, 2, 2, 0, None, 0, None, 0, stream())
    assert rc == -2 and b"multiples of 8" in lib.b200_last_error()


# ------------------------------------------------------------------ conv
@pytest.mark.parametrize("N,C,H,O,k,s,p,res,relu", [
    (2, 8, 56, 64, 7, 2, 3, False, True),     # stem after channel padding 3 -> 8
    (3, 8, 224, 64, 7, 2, 3, False, True),    # full-size stem: several output rows per CTA, image borders inside a CTA's rows
    (20, 8, 64, 48, 7, 2, 3, False, False),   # stem with fewer than 64 output channels, no ReLU
    (1, 64, 56, 64, 3, 1, 1, True, True),
    (2, 64, 56, 128, 3, 2, 1, False, True),
    (2, 64, 56, 128, 1, 2, 0, False, False),
    (3, 256, 14, 1024, 1, 1, 0, True, True),
    (1, 512, 7, 512, 3, 1, 1, False, True),
    (8, 64, 56, 64, 3, 1, 1, True, True),      # enough tiles for the persistent kernel, tiles cross image borders
    (32, 64, 56, 128, 3, 2, 1, False, True),   # persistent, stride 2
    (5, 128, 28, 128, 3, 1, 1, False, False),  # odd image count: the last tile runs past the tensor
    (16, 64, 56, 64, 3, 1, 1, False, True),    # several tiles per CTA: the 72 KB weight tile stays resident in shared memory
    (16, 64, 56, 512, 1, 1, 0, True, True),    # resident weights, two 256-wide column tiles: the weight tile is replaced mid-kernel
    (16, 128, 28, 256, 1, 1, 0, True, True),   # 128-wide tiles, two column tiles, residual
    (52, 256, 28, 64, 1, 1, 0, False, False),  # resident weights with four k-blocks per tile, ragged last tile
    (41, 128, 28, 512, 1, 1, 0, True, True),   # column tiles fastest: each CTA keeps one of four column tiles, ragged last row tile
    (1, 64, 56, 256, 1, 1, 0, True, True),     # few tiles, nothing to split: one k-block, the staged epilogue
    (1, 2048, 7, 512, 1, 1, 0, False, True),   # few tiles, taps split eight ways (four k-blocks each), 49 rows
    (2, 512, 14, 512, 3, 2, 1, False, True),   # 72 k-blocks over eight CTAs: a split starts inside a filter tap
    (3, 192, 9, 72, 3, 2, 1, True, False),     # 27 k-blocks in uneven splits, output channels past a whole tile
    (1, 128, 56, 130, 1, 2, 0, False, True),   # output rows without 8-byte alignment
    (1, 64, 40, 64, 3, 9, 1, False, True),     # no im2col map (stride past 8): threads gather the pixels; one tile
    (2, 192, 100, 200, 3, 9, 1, True, True),   # the same, several ragged tiles, 27 k-blocks, residual
    (1, 64, 6, 64, 3, 1, 128, False, False),   # no im2col map (padding past 127) and a tile for every SM: the persistent kernel gathers
    (1, 64, 6, 136, 1, 1, 128, True, True),    # the same, two column tiles, residual
    (37, 256, 14, 1024, 1, 1, 0, True, False), # column tiles fastest with eight column tiles (grid trimmed to a multiple of 8)
])
def test_conv2d_nhwc(lib, N, C, H, O, k, s, p, res, relu):
    dtype = torch.float16
    x = gen((N, C, H, H), dtype)
    w = gen((O, C, k, k), torch.float32, 1, math.sqrt(2.0 / (C * k * k)))
    gamma, beta = torch.rand(O) + 0.5, torch.randn(O) * 0.1
    mean, var = torch.randn(O) * 0.1, torch.rand(O) + 0.5
    Ho = (H + 2 * p - k) // s + 1
    r = gen((N, O, Ho, Ho), dtype, 5) if res else None
    ref = torch.nn.functional.conv2d(x.float(), w, None, s, p)
    ref = torch.nn.functional.batch_norm(ref, mean, var, gamma, beta, False, 0.0, 1e-5)
    if res:
        ref = ref + r.float()
    if relu:
        ref = torch.relu(ref)
    xd = x.cuda().contiguous(memory_format=torch.channels_last)
    wd = torch.empty(O * k * k * C, dtype=dtype, device="cuda")
    bd = torch.empty(O, dtype=torch.float32, device="cuda")
    prm = [t.cuda() for t in (gamma, beta, mean, var)]
    wc = w.cuda()
    ok(lib, lib.b200_conv_weight_prep(wc.data_ptr(), None, *[t.data_ptr() for t in prm], wd.data_ptr(), bd.data_ptr(), O, C, k, k, C,
                                      1e-5, 0, 0, 1, stream()))
    y = torch.empty(N, O, Ho, Ho, dtype=dtype, device="cuda").contiguous(memory_format=torch.channels_last)
    rd = r.cuda().contiguous(memory_format=torch.channels_last) if res else None
    ok(lib, lib.b200_conv2d_nhwc(xd.data_ptr(), wd.data_ptr(), bd.data_ptr(), rd.data_ptr() if res else None, y.data_ptr(), N, H, H, C, C,
                                 O, k, k, s, s, p, p, Ho, Ho, 1, 1 if relu else 0, stream()))
    close(y, ref, rtol=2e-2, atol=3e-2)


# ------------------------------------------------------------------ attention
def attn_ref(q, k, v, mask, scale, dtype):
    G = q.shape[1] // k.shape[1]
    k, v = k.float().repeat_interleave(G, 1), v.float().repeat_interleave(G, 1)
    s = q.float() @ k.transpose(-1, -2) * scale
    if mask is not None:
        s = s + mask.float()
    return torch.softmax(s, -1) @ v


@pytest.mark.parametrize("B,S,valid", [(1, 4352, 4097), (8, 4352, 4100), (3, 80, 37), (2, 272, 272), (64, 512, 300), (64, 4352, 4097), (5, 8192, 6000)])
def test_attn_decode(lib, B, S, valid):
    import model_zoo as mz

    dtype, Hq, Hkv, D = torch.bfloat16, 12, 2, 128
    q, k, v = gen((B, Hq, 1, D), dtype), gen((B, Hkv, S, D), dtype, 1), gen((B, Hkv, S, D), dtype, 2)
    mask = mz.causal_mask(B, 1, S, valid - 1)
    ref = attn_ref(q, k, v, mask, D ** -0.5, dtype)[:, :, 0]
    Q, K, V, M = q.cuda(), k.cuda(), v.cuda(), mask.cuda()
    out = torch.empty(B, Hq, D, dtype=dtype, device="cuda")
    ws = torch.empty(lib.b200_attn_decode_workspace_bytes(B, Hq, Hkv, S, D), dtype=torch.uint8, device="cuda")
    ok(lib, lib.b200_attn_decode(Q.data_ptr(), K.data_ptr(), V.data_ptr(), M.data_ptr(), out.data_ptr(), B, Hq, Hkv, S, D, Hq * D,
                                 Hkv * S * D, S * D, S, D ** -0.5, 2, ws.data_ptr(), ws.numel(), stream()))
    close(out, ref, rtol=2e-2, atol=5e-3)
    # no mask = attend to everything
    ok(lib, lib.b200_attn_decode(Q.data_ptr(), K.data_ptr(), V.data_ptr(), None, out.data_ptr(), B, Hq, Hkv, S, D, Hq * D,
                                 Hkv * S * D, S * D, 0, D ** -0.5, 2, ws.data_ptr(), ws.numel(), stream()))
    close(out, attn_ref(q, k, v, None, D ** -0.5, dtype)[:, :, 0], rtol=2e-2, atol=5e-3)


@pytest.mark.parametrize("B,S,valid,shift", [(1, 32768, 20001, 0), (1, 32768, 32768, 1), (2, 17000, 1, 0), (3, 448, 447, 0), (1, 16, 5, 1), (1, 64, 64, 0),
                                             (64, 448, 300, 0), (7, 17000, 9000, 1), (6, 17000, 17000, 0), (40, 300, 299, 1)])
def test_attn_decode_merge_of_workspace_partials(lib, B, S, valid, shift):
    """Caches outside 512..16384 rows leave their splits' partial sums in the workspace for a second kernel: one
    split, fewer splits than the kernel has groups, 256 of them with the masked ones empty; many heads with few and
    with many splits; a workspace that is only 4-byte aligned."""
    import model_zoo as mz

    dtype, Hq, Hkv, D = torch.bfloat16, 12, 2, 128
    q, k, v = gen((B, Hq, 1, D), dtype), gen((B, Hkv, S, D), dtype, 1), gen((B, Hkv, S, D), dtype, 2)
    mask = mz.causal_mask(B, 1, S, valid - 1)
    ref = attn_ref(q, k, v, mask, D ** -0.5, dtype)[:, :, 0]
    Q, K, V, M = q.cuda(), k.cuda(), v.cuda(), mask.cuda()
    out = torch.empty(B, Hq, D, dtype=dtype, device="cuda")
    need = lib.b200_attn_decode_workspace_bytes(B, Hq, Hkv, S, D)
    assert need > 0
    ws = torch.full((need // 4 + 1,), float("nan"), device="cuda")[shift:]   # every partial that is read has been written
    ok(lib, lib.b200_attn_decode(Q.data_ptr(), K.data_ptr(), V.data_ptr(), M.data_ptr(), out.data_ptr(), B, Hq, Hkv, S, D, Hq * D,
                                 Hkv * S * D, S * D, S, D ** -0.5, 2, ws.data_ptr(), need, stream()))
    close(out, ref, rtol=2e-2, atol=5e-3)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("B", [2, 12])
def test_attn_decode_small_batches_in_both_dtypes(lib, dtype, B):
    """Small batches take clusters of 16 splits (a non-portable cluster size that every kernel instantiation has to
    be allowed separately), B=12 the portable eight: both activation types, in one process, against the fp32 reference."""
    import model_zoo as mz

    S, valid, Hq, Hkv, D = 1024, 700, 12, 2, 128
    q, k, v = gen((B, Hq, 1, D), dtype), gen((B, Hkv, S, D), dtype, 1), gen((B, Hkv, S, D), dtype, 2)
    mask = mz.causal_mask(B, 1, S, valid - 1).to(dtype)
    ref = attn_ref(q, k, v, mask, D ** -0.5, dtype)[:, :, 0]
    Q, K, V, M = q.cuda(), k.cuda(), v.cuda(), mask.cuda()
    out = torch.empty(B, Hq, D, dtype=dtype, device="cuda")
    ws = torch.empty(max(16, lib.b200_attn_decode_workspace_bytes(B, Hq, Hkv, S, D)), dtype=torch.uint8, device="cuda")
    code = 2 if dtype == torch.bfloat16 else 1
    ok(lib, lib.b200_attn_decode(Q.data_ptr(), K.data_ptr(), V.data_ptr(), M.data_ptr(), out.data_ptr(), B, Hq, Hkv, S, D, Hq * D,
                                 Hkv * S * D, S * D, S, D ** -0.5, code, ws.data_ptr(), ws.numel(), stream()))
    close(out, ref, rtol=2e-2, atol=5e-3)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("Hq,Hkv", [(12, 2), (7, 7), (8, 1)])
@pytest.mark.parametrize("B,S", [(1, 1024), (1, 1040), (3, 1111), (3, 1536), (3, 1800), (1, 4352), (4, 2048), (1, 16383)])
def test_attn_decode_eight_warps(lib, dtype, Hq, Hkv, B, S):
    """Few sequences with more than 64 or 96 keys per split take eight warps per CTA: on both sides of that line and of the number
    of clusters that fit, masks with a filled prefix, with holes, with one key; against float64 within the rounding
    of probabilities and outputs (2^-8 of what is added up in bf16, 2^-11 in fp16; fp32 elsewhere)."""
    D, neg = 128, torch.finfo(dtype).min
    q, k, v = gen((B, Hq, 1, D), dtype), gen((B, Hkv, S, D), dtype, 1), gen((B, Hkv, S, D), dtype, 2)
    g = torch.Generator().manual_seed(S)
    mask = torch.zeros(B, 1, 1, S)
    mask[0, ..., (3 * S) // 4:] = neg
    if B > 1:
        mask[1] = torch.where(torch.rand(S, generator=g) < 0.3, 0.0, neg)
    if B > 2:
        mask[2] = neg
        mask[2, ..., S - 1] = 0
    mask = mask.to(dtype)
    s = (q.double() @ k.double().repeat_interleave(Hq // Hkv, 1).transpose(2, 3)) * D ** -0.5 + mask.double()
    p, vd = s.softmax(-1), v.double().repeat_interleave(Hq // Hkv, 1)
    want, size = (p @ vd)[:, :, 0], (p @ vd.abs())[:, :, 0]
    Q, K, V, M = q.cuda(), k.cuda(), v.cuda(), mask.cuda()
    out = torch.full((B, Hq, D), float("nan"), dtype=dtype, device="cuda")
    ok(lib, lib.b200_attn_decode(Q.data_ptr(), K.data_ptr(), V.data_ptr(), M.data_ptr(), out.data_ptr(), B, Hq, Hkv, S, D, Hq * D,
                                 Hkv * S * D, S * D, S, D ** -0.5, DT[dtype], None, 0, stream()))
    eps = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    err = (out.double().cpu() - want).abs()
    assert (err <= (size + want.abs()) * eps * 1.01 + 1e-5).all(), float(err.max())


@pytest.mark.parametrize("B,S,Hq,Hkv", [(40, 2048, 12, 2), (64, 4352, 12, 2), (33, 1000, 8, 1), (130, 640, 4, 4)])
def test_attn_decode_many_sequences_ragged_masks(lib, B, S, Hq, Hkv):
    """Batches large enough for the balanced kernel (every CTA gets the same number of unmasked 16-key
    blocks): each sequence has its own attended length - from a single key to the whole cache - some
    masks have holes, and the call is repeated (the tickets of the merge must return to zero)."""
    dtype, D = torch.bfloat16, 128
    g = torch.Generator().manual_seed(B)
    q, k, v = gen((B, Hq, 1, D), dtype), gen((B, Hkv, S, D), dtype, 1), gen((B, Hkv, S, D), dtype, 2)
    neg = torch.finfo(dtype).min
    mask = torch.full((B, 1, 1, S), neg, dtype=dtype)
    lengths = torch.randint(1, S + 1, (B,), generator=g)
    lengths[0], lengths[1], lengths[2] = 1, S, 17
    for b in range(B):
        mask[b, 0, 0, :lengths[b]] = 0
        if b % 5 == 3 and lengths[b] > 200:      # a hole of masked keys inside the attended range
            mask[b, 0, 0, 64:160] = neg
        if b % 7 == 4:
            mask[b, 0, 0, :lengths[b]] = torch.where(torch.rand(int(lengths[b]), generator=g) < 0.5, 0.0, neg).to(dtype)
            mask[b, 0, 0, 0] = 0
    ref = attn_ref(q, k, v, mask, D ** -0.5, dtype)[:, :, 0]
    Q, K, V, M = q.cuda(), k.cuda(), v.cuda(), mask.cuda()
    ws = torch.empty(max(16, lib.b200_attn_decode_workspace_bytes(B, Hq, Hkv, S, D)), dtype=torch.uint8, device="cuda")
    for _ in range(2):
        out = torch.full((B, Hq, D), float("nan"), dtype=dtype, device="cuda")
        ok(lib, lib.b200_attn_decode(Q.data_ptr(), K.data_ptr(), V.data_ptr(), M.data_ptr(), out.data_ptr(), B, Hq, Hkv, S, D, Hq * D,
                                     Hkv * S * D, S * D, S, D ** -0.5, 2, ws.data_ptr(), ws.numel(), stream()))
        close(out, ref, rtol=2e-2, atol=5e-3)
    # a sequence whose mask admits no key gives zeros (ATen would average all rows; no model produces such a mask)
    mask[5] = neg
    out = torch.full((B, Hq, D), float("nan"), dtype=dtype, device="cuda")
    ok(lib, lib.b200_attn_decode(Q.data_ptr(), K.data_ptr(), V.data_ptr(), mask.cuda().data_ptr(), out.data_ptr(), B, Hq, Hkv, S, D, Hq * D,
                                 Hkv * S * D, S * D, S, D ** -0.5, 2, ws.data_ptr(), ws.numel(), stream()))
    assert (out[5] == 0).all()
    keep = [b for b in range(B) if b != 5]
    close(out[keep], ref[keep], rtol=2e-2, atol=5e-3)


@pytest.mark.parametrize("B,T", [(1, 512), (2, 48), (1, 100), (1, 2048), (2, 328)])
def test_attn_prefill(lib, B, T):
    import model_zoo as mz

    dtype, Hq, Hkv, D = torch.bfloat16, 12, 2, 128
    q = gen((B, T, Hq, D), dtype).transpose(1, 2)          # the layout the graph produces: a transposed view
    k, v = gen((B, Hkv, T, D), dtype, 1), gen((B, T, Hkv, D), dtype, 2).transpose(1, 2)
    mask = mz.causal_mask(1, T, T, 0)
    ref = attn_ref(q, k, v, mask, D ** -0.5, dtype).transpose(1, 2)
    Q, K, V, M = (t.cuda() for t in (q.transpose(1, 2).contiguous(), k, v.transpose(1, 2).contiguous(), mask))
    Q, V = Q.transpose(1, 2), V.transpose(1, 2)
    out = torch.full((B, T, Hq, D), float("nan"), dtype=dtype, device="cuda")
    st = lambda t: (C.c_int64 * 3)(*t.stride()[:3])
    ok(lib, lib.b200_attn_prefill(Q.data_ptr(), K.data_ptr(), V.data_ptr(), M.data_ptr(), out.data_ptr(), B, Hq, Hkv, T, T, D,
                                  st(Q), st(K), st(V), 0, T, D ** -0.5, 2, stream()))
    close(out, ref, rtol=2e-2, atol=5e-3)
    code = C.c_int(0)
    ok(lib, lib.b200_debug_device_error(C.byref(code), 1))
    assert code.value == 0


@pytest.mark.parametrize("B,T,aligned", [(1, 777, True), (2, 100, "shared"), (1, 777, False), (2, 33, True), (1, 129, True), (1, 65, True)])
def test_attn_prefill_ragged_lengths(lib, B, T, aligned):
    """Lengths that are no multiple of eight: mask rows padded to 16 bytes (the tensor-map kernel; the padding is NaN and
    must not be read as a mask) and dense rows (the mma.sync kernel)."""
    import model_zoo as mz

    dtype, Hq, Hkv, D = torch.bfloat16, 4, 2, 128
    q, k, v = gen((B, Hq, T, D), dtype), gen((B, Hkv, T, D), dtype, 1), gen((B, Hkv, T, D), dtype, 2)
    shared = aligned == "shared"   # one mask for all sequences: a batch stride of zero
    mask = mz.causal_mask(1 if shared else B, T, T, 0)
    Tp = -(-T // 8) * 8 if aligned else T
    M = torch.full((1 if shared else B, 1, T, Tp), float("nan"), dtype=dtype, device="cuda")
    M[..., :T] = mask.cuda()
    Q, K, V = q.cuda(), k.cuda(), v.cuda()
    out = torch.full((B, T, Hq, D), float("nan"), dtype=dtype, device="cuda")
    st = lambda t: (C.c_int64 * 3)(*t.stride()[:3])
    ok(lib, lib.b200_attn_prefill(Q.data_ptr(), K.data_ptr(), V.data_ptr(), M.data_ptr(), out.data_ptr(), B, Hq, Hkv, T, T, D,
                                  st(Q), st(K), st(V), 0 if shared else T * Tp, Tp, D ** -0.5, 2, stream()))
    close(out, attn_ref(q, k, v, mask, D ** -0.5, dtype).transpose(1, 2), rtol=2e-2, atol=5e-3)


@pytest.mark.parametrize("S", [64, 128, 192, 2048, 4032])
@pytest.mark.parametrize("slow", [0, 1, 2, 3])
def test_attn_prefill_row_quarters_out_of_step(lib, slow, S):
    """The four groups of 32 query rows that share a tile are not kept in step: here one of them has to rescale its sums
    in every key tile (its scores rise along the keys) and the others never (their largest score is the first key's), so
    that they run ahead by as much as the barriers let them.  The bound: probabilities and outputs rounded to bf16
    (eight significant bits: 2^-8 of the magnitudes that are added up, and of the result), the rest is fp32."""
    dtype, B, Hq, Hkv, T, D = torch.bfloat16, 1, 16, 4, 128, 128
    q, k, v = gen((B, Hq, T, D), dtype, 0, 0.3), gen((B, Hkv, S, D), dtype, 1, 0.3), gen((B, Hkv, S, D), dtype, 2)
    rows = torch.arange(T) // 32 == slow
    q[..., :2] = 0
    q[:, :, rows, 0] = 8.0
    q[:, :, ~rows, 1] = 8.0
    k[..., 0] = (torch.arange(S) // 64) * 0.25      # + 0.18 per key tile in the exponent
    k[..., 1] = 0
    k[:, :, 0, 1] = 6.0                             # 4.2 above the others
    Q, K, V = q.cuda(), k.cuda(), v.cuda()
    st = lambda t: (C.c_int64 * 3)(*t.stride()[:3])
    s = (q.double() @ k.double().repeat_interleave(Hq // Hkv, 1).transpose(2, 3)) * D ** -0.5
    p = s.softmax(-1)
    vd = v.double().repeat_interleave(Hq // Hkv, 1)
    want, size = (p @ vd).transpose(1, 2), (p @ vd.abs()).transpose(1, 2)
    for _ in range(3):
        out = torch.full((B, T, Hq, D), float("nan"), dtype=dtype, device="cuda")
        ok(lib, lib.b200_attn_prefill(Q.data_ptr(), K.data_ptr(), V.data_ptr(), None, out.data_ptr(), B, Hq, Hkv, T, S, D,
                                      st(Q), st(K), st(V), 0, 0, D ** -0.5, 2, stream()))
        err = (out.double().cpu() - want).abs()
        assert (err <= (size + want.abs()) * 2.0 ** -8 * 1.01 + 1e-5).all(), float(err.max())


def _mask_of(kind, B, T, S, dtype):
    """[B, T, S] additive masks: all, some or none of the 128 x 128 tiles are masked, zero or mixed."""
    neg = torch.finfo(dtype).min
    r, c = torch.arange(T)[:, None], torch.arange(S)[None]
    m = torch.zeros(B, T, S)
    if kind == "causal":
        m[:] = torch.where(c <= r + S - T, 0.0, neg)
    elif kind == "bias":             # finite values everywhere
        m[:] = -0.02 * (r - c).abs()
    elif kind == "holes":            # whole tiles masked, rows without any key, a tile with one key, infinities
        m[:, :, 128:256] = neg
        m[:, : T // 2, 256:384] = float("-inf")
        m[:, T // 3, :] = neg
        m[0, T - 1, 200 % S] = 0
    elif kind == "late":             # the first key tile (and more) is not wanted
        m[:, :, : min(S - 1, 300)] = neg
    elif kind == "first":            # only the first key tile; the last sequence sees everything but the last key
        m[:, :, 128:] = neg
        m[-1, :, :] = 0
        m[-1, :, S - 1:] = neg
    return m.to(dtype)


@pytest.mark.parametrize("kind", ["causal", "bias", "holes", "first", "late"])
@pytest.mark.parametrize("B,T,S", [(1, 1, 128), (1, 2, 129), (2, 127, 255), (1, 128, 1), (2, 129, 384), (1, 300, 640), (1, 64, 1111)])
@pytest.mark.parametrize("rows", ["aligned", "dense", "shared", "one row"])
def test_attn_prefill_mask_tiles(lib, kind, B, T, S, rows):
    """Mask tiles that are masked, zero or mixed, in every form of addressing, with the states found beforehand and by the
    kernel itself: both equal float64 within the rounding of probabilities and outputs to bf16 (2^-8 of what is added up,
    fp32 elsewhere), and rows that attend to nothing give zeros."""
    dtype, Hq, Hkv, D = torch.bfloat16, 4, 2, 128
    q, k, v = gen((B, Hq, T, D), dtype), gen((B, Hkv, S, D), dtype, 1), gen((B, Hkv, S, D), dtype, 2)
    mask = _mask_of(kind, B, T, S, dtype)
    pitch = -(-S // 8) * 8 if rows == "aligned" else S
    if rows == "shared":
        mask = mask[-1:]
    if rows == "one row":
        mask = mask[:, -1:]
    M = torch.full((mask.shape[0], mask.shape[1], pitch), float("nan"), dtype=dtype, device="cuda")
    M[..., :S] = mask.cuda()
    mb, mt = (0 if rows == "shared" else M.stride(0)), (0 if rows == "one row" else pitch)
    nb = 1 if rows == "shared" else B
    tiles = torch.full((nb, -(-T // 128), -(-S // 128)), 9, dtype=torch.uint8, device="cuda")
    ok(lib, lib.b200_mask_tiles(M.data_ptr(), nb, T, S, mb, mt, 2, tiles.data_ptr(), stream()))
    full = mask.double().expand(B, T, S)
    for i in range(tiles.shape[1]):
        for j in range(tiles.shape[2]):
            t = full[:nb, i * 128:(i + 1) * 128, j * 128:(j + 1) * 128].flatten(1)
            want = torch.where((t > -1e30).any(1), torch.where((t == 0).all(1), 1, 2), 0)
            assert tiles[:, i, j].tolist() == want.tolist(), (i, j)
    s = (q.double() @ k.double().repeat_interleave(Hq // Hkv, 1).transpose(2, 3)) * D ** -0.5 + full[:, None].clamp(min=-1e300)
    dead = (full <= -1e30).all(-1)
    p = s.softmax(-1) * ~dead[:, None, :, None]
    vd = v.double().repeat_interleave(Hq // Hkv, 1)
    want, size = (p @ vd).transpose(1, 2), (p @ vd.abs()).transpose(1, 2)
    Q, K, V = q.cuda(), k.cuda(), v.cuda()
    st = lambda t: (C.c_int64 * 3)(*t.stride()[:3])
    got = []
    for states in (None, tiles.data_ptr()):
        out = torch.full((B, T, Hq, D), float("nan"), dtype=dtype, device="cuda")
        ok(lib, lib.b200_attn_prefill_tiles(Q.data_ptr(), K.data_ptr(), V.data_ptr(), M.data_ptr(), states, out.data_ptr(), B, Hq, Hkv, T, S, D,
                                            st(Q), st(K), st(V), mb, mt, D ** -0.5, 2, stream()))
        err = (out.double().cpu() - want).abs()
        assert (err <= (size + want.abs()) * 2.0 ** -8 * 1.01 + 1e-5).all(), float(err.max())
        got.append(out)
    assert torch.equal(*got)
    code = C.c_int(0)
    ok(lib, lib.b200_debug_device_error(C.byref(code), 1))
    assert code.value == 0


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("kind", [None, "causal", "bias", "last"])
@pytest.mark.parametrize("B,T,S", [(1, 1, 1), (2, 5, 7), (1, 16, 16), (3, 17, 17), (1, 63, 63), (2, 64, 64), (1, 65, 64), (2, 130, 33), (1, 3, 64), (1, 20, 65)])
def test_attn_prefill_few_keys(lib, B, T, S, kind, dtype):
    """Up to 64 keys are one tile of the mma.sync kernel, whose mask rows are copied to the last key and no further (what lies
    behind is no number here).  Bound: probabilities and outputs rounded to the activation type, of what is added up."""
    Hq, Hkv, D = 4, 2, 128
    q, k, v = gen((B, Hq, T, D), dtype), gen((B, Hkv, S, D), dtype, 1), gen((B, Hkv, S, D), dtype, 2)
    mask = torch.zeros(B, T, S).to(dtype)
    if kind == "last":   # one key each
        mask[:] = torch.finfo(dtype).min
        mask[..., S - 1] = 0
    elif kind:
        mask = _mask_of(kind, B, T, S, dtype)
        if kind == "causal" and dtype == torch.float16:
            # a row of nothing but fp16's lowest value (-65504) keeps its scores to a half unit of fp32 there, 2^-9: half a per cent of each probability
            mask[:, :max(T - S, 0), 0] = 0
    s = (q.double() @ k.double().repeat_interleave(Hq // Hkv, 1).transpose(2, 3)) * D ** -0.5 + mask.double()[:, None]
    p = s.softmax(-1) * ~(mask.double() <= -1e30).all(-1)[:, None, :, None]
    vd = v.double().repeat_interleave(Hq // Hkv, 1)
    want, size = (p @ vd).transpose(1, 2), (p @ vd.abs()).transpose(1, 2)
    pitch = -(-S // 8) * 8
    M = torch.full((B, T, pitch), float("nan"), dtype=dtype, device="cuda")
    M[..., :S] = mask.cuda()
    Q, K, V = q.cuda(), k.cuda(), v.cuda()
    st = lambda t: (C.c_int64 * 3)(*t.stride()[:3])
    out = torch.full((B, T, Hq, D), float("nan"), dtype=dtype, device="cuda")
    ok(lib, lib.b200_attn_prefill(Q.data_ptr(), K.data_ptr(), V.data_ptr(), M.data_ptr() if kind else None, out.data_ptr(), B, Hq, Hkv, T, S, D, st(Q), st(K), st(V),
                                  T * pitch, pitch, D ** -0.5, DT[dtype], stream()))
    eps = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    err = (out.double().cpu() - want).abs()
    assert (err <= (size + want.abs()) * eps * 1.01 + 1e-5).all(), float(err.max())


@pytest.mark.parametrize("T,S,kernel", [(16, 16, "attn_prefill_kernel"), (200, 64, "attn_prefill_kernel"), (3, 65, "attn_prefill_tc5_kernel"), (129, 100, "attn_prefill_tc5_kernel")])
def test_attn_prefill_runs_on_the_kernel_that_its_keys_call_for(lib, T, S, kernel):
    Q, K = torch.zeros(1, 4, T, 128, dtype=torch.bfloat16, device="cuda"), torch.zeros(1, 2, S, 128, dtype=torch.bfloat16, device="cuda")
    out = torch.empty(1, T, 4, 128, dtype=torch.bfloat16, device="cuda")
    st = lambda t: (C.c_int64 * 3)(*t.stride()[:3])
    names = kernels_of(lambda: go(lib, lib.b200_attn_prefill(Q.data_ptr(), K.data_ptr(), K.data_ptr(), None, out.data_ptr(), 1, 4, 2, T, S, 128, st(Q), st(K), st(K),
                                                             0, 0, 0.1, 2, stream())))
    assert len(names) == 1 and kernel + "<" in names[0], names


@pytest.mark.parametrize("T", [128, 400])
def test_attn_prefill_many_launches_in_a_row(lib, T):
    """The first key tile is requested before it is known to be wanted, so its scores may be complete before the producer
    looks at the stage again: a few hundred launches, all equal, no wait that runs out."""
    dtype, Hq, Hkv, D = torch.bfloat16, 12, 2, 128
    Q, K, V = gen((1, Hq, T, D), dtype).cuda(), gen((1, Hkv, T, D), dtype, 1).cuda(), gen((1, Hkv, T, D), dtype, 2).cuda()
    M = _mask_of("causal", 1, T, T, dtype).cuda()
    tiles = torch.empty(1, -(-T // 128), -(-T // 128), dtype=torch.uint8, device="cuda")
    ok(lib, lib.b200_mask_tiles(M.data_ptr(), 1, T, T, 0, T, 2, tiles.data_ptr(), stream()))
    st = lambda t: (C.c_int64 * 3)(*t.stride()[:3])
    outs = [torch.empty((1, T, Hq, D), dtype=dtype, device="cuda") for _ in range(200)]
    for out in outs:
        go(lib, lib.b200_attn_prefill_tiles(Q.data_ptr(), K.data_ptr(), V.data_ptr(), M.data_ptr(), tiles.data_ptr(), out.data_ptr(), 1, Hq, Hkv,
                                            T, T, D, st(Q), st(K), st(V), 0, T, D ** -0.5, 2, stream()))
    assert all(torch.equal(outs[0], out) for out in outs[1:])
    code = C.c_int(0)
    ok(lib, lib.b200_debug_device_error(C.byref(code), 1))
    assert code.value == 0


@pytest.mark.parametrize("lead", [64, 128, 1000, 3000])
def test_attn_prefill_first_key_tiles_masked_and_keys_far_away(lib, lead):
    """The first key tile is requested before the mask is known.  Where it is not wanted its copies, from memory that no cache
    holds, may be the last thing to arrive: nobody may take them for the first tile that is.  Launch after launch over
    caches that together outgrow the L2: equal to a launch whose operands are at hand, and to float64."""
    dtype, B, T, S, Hq, Hkv, D, sets = torch.bfloat16, 8, 16, 4096, 12, 2, 128, 5
    mask = torch.zeros(1, T, S).to(dtype)
    mask[..., :lead] = torch.finfo(dtype).min
    Q, M = gen((B, Hq, T, D), dtype).cuda(), mask.cuda()
    K = [gen((B, Hkv, S, D), dtype, 1 + i).cuda() for i in range(sets)]
    V = [gen((B, Hkv, S, D), dtype, 9 + i).cuda() for i in range(sets)]
    tiles = torch.empty(1, 1, S // 128, dtype=torch.uint8, device="cuda")
    ok(lib, lib.b200_mask_tiles(M.data_ptr(), 1, T, S, 0, S, 2, tiles.data_ptr(), stream()))
    st = lambda t: (C.c_int64 * 3)(*t.stride()[:3])

    def call(i):
        out = torch.full((B, T, Hq, D), float("nan"), dtype=dtype, device="cuda")
        go(lib, lib.b200_attn_prefill_tiles(Q.data_ptr(), K[i].data_ptr(), V[i].data_ptr(), M.data_ptr(), tiles.data_ptr(), out.data_ptr(), B, Hq, Hkv,
                                            T, S, D, st(Q), st(K[i]), st(V[i]), 0, S, D ** -0.5, 2, stream()))
        return out

    cold = [[call(i) for i in range(sets)] for _ in range(8)]
    for i in range(sets):
        call(i)
        warm = call(i)
        assert all(torch.equal(warm, c[i]) for c in cold)
        p = ((Q.double() @ K[i][:, :, lead:].double().repeat_interleave(6, 1).transpose(2, 3)) * D ** -0.5).softmax(-1)
        vd = V[i][:, :, lead:].double().repeat_interleave(6, 1)
        want, size = (p @ vd).transpose(1, 2), (p @ vd.abs()).transpose(1, 2)
        assert ((warm.double() - want).abs() <= (size + want.abs()) * 2.0 ** -8 * 1.01 + 1e-5).all()
    code = C.c_int(0)
    ok(lib, lib.b200_debug_device_error(C.byref(code), 1))
    assert code.value == 0


@pytest.mark.parametrize("scale", [0.0, -0.07])
@pytest.mark.parametrize("S", [60, 100, 129, 200, 256])
@pytest.mark.parametrize("masked", [None, "zero", "causal"])
def test_attn_prefill_scales_that_are_not_positive(lib, masked, S, scale):
    """Scale 0 weighs all keys alike and a negative one turns their order round, also where the last key tile, or half of it,
    lies past the end.  Bound as for any mask: 2^-8 of what is added up."""
    dtype, Hq, Hkv, D, T = torch.bfloat16, 4, 2, 128, 130
    q, k, v = gen((1, Hq, T, D), dtype), gen((1, Hkv, S, D), dtype, 1), gen((1, Hkv, S, D), dtype, 2)
    mask = torch.zeros(1, T, S).to(dtype) if masked == "zero" else _mask_of("causal", 1, T, S, dtype) if masked else None
    s = (q.double() @ k.double().repeat_interleave(2, 1).transpose(2, 3)) * scale + (mask.double()[:, None] if masked else 0)
    dead = (mask.double() <= -1e30).all(-1)[:, None, :, None] if masked else torch.zeros((), dtype=torch.bool)
    p, vd = s.softmax(-1) * ~dead, v.double().repeat_interleave(2, 1)
    want, size = (p @ vd).transpose(1, 2), (p @ vd.abs()).transpose(1, 2)
    pitch = -(-S // 8) * 8
    Q, K, V, M = q.cuda(), k.cuda(), v.cuda(), torch.zeros(1, T, pitch, dtype=dtype, device="cuda")
    if masked:
        M[..., :S] = mask.cuda()
    st = lambda t: (C.c_int64 * 3)(*t.stride()[:3])
    out = torch.full((1, T, Hq, D), float("nan"), dtype=dtype, device="cuda")
    ok(lib, lib.b200_attn_prefill(Q.data_ptr(), K.data_ptr(), V.data_ptr(), M.data_ptr() if masked else None, out.data_ptr(), 1, Hq, Hkv, T, S, D,
                                  st(Q), st(K), st(V), 0, pitch if masked else 0, scale, 2, stream()))
    err = (out.double().cpu() - want).abs()
    assert (err <= (size + want.abs()) * 2.0 ** -8 * 1.01 + 1e-5).all(), float(err.max())


@pytest.mark.parametrize("known", [True, False])
def test_attn_prefill_row_blocks_without_keys(lib, known):
    """Blocks of 128 rows whose mask admits no key have only their copies to wait for: next to blocks that work, and in
    launches that follow at once and use the same shared memory, with states found beforehand and by the kernel itself."""
    dtype, Hq, Hkv, D, T, S = torch.bfloat16, 12, 2, 128, 1700, 300
    q, k, v = gen((1, Hq, T, D), dtype), gen((1, Hkv, S, D), dtype, 1), gen((1, Hkv, S, D), dtype, 2)
    mask = torch.full((1, T, 304), torch.finfo(dtype).min, dtype=dtype)
    mask[:, 128 * 3:128 * 5, :S] = 0
    Q, K, V, M = q.cuda(), k.cuda(), v.cuda(), mask.cuda()
    tiles = torch.empty(1, -(-T // 128), -(-S // 128), dtype=torch.uint8, device="cuda")
    ok(lib, lib.b200_mask_tiles(M.data_ptr(), 1, T, S, 0, 304, 2, tiles.data_ptr(), stream()))
    st = lambda t: (C.c_int64 * 3)(*t.stride()[:3])
    outs = [torch.full((1, T, Hq, D), float("nan"), dtype=dtype, device="cuda") for _ in range(50)]
    for out in outs:
        go(lib, lib.b200_attn_prefill_tiles(Q.data_ptr(), K.data_ptr(), V.data_ptr(), M.data_ptr(), tiles.data_ptr() if known else None, out.data_ptr(), 1, Hq, Hkv,
                                            T, S, D, st(Q), st(K), st(V), 0, 304, D ** -0.5, 2, stream()))
    rows = slice(128 * 3, 128 * 5)
    p = ((q[:, :, rows].double() @ k.double().repeat_interleave(6, 1).transpose(2, 3)) * D ** -0.5).softmax(-1)
    vd = v.double().repeat_interleave(6, 1)
    want, size = (p @ vd).transpose(1, 2), (p @ vd.abs()).transpose(1, 2)
    for out in outs:
        got = out.double().cpu()
        assert ((got[:, rows] - want).abs() <= (size + want.abs()) * 2.0 ** -8 * 1.01 + 1e-5).all()
        got[:, rows] = 0
        assert not got.any()
    code = C.c_int(0)
    ok(lib, lib.b200_debug_device_error(C.byref(code), 1))
    assert code.value == 0


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_attn_prefill_arbitrary_masks_and_no_mask(lib, dtype):
    """Nothing in the kernels assumes a causal mask: a per-sequence mask with windows, holes and key
    tiles that are masked for a whole block of query rows (those tiles are skipped), S != T, and no
    mask at all."""
    B, T, S, Hq, Hkv, D = 2, 200, 456, 4, 2, 128
    g = torch.Generator().manual_seed(11)
    q, k, v = gen((B, Hq, T, D), dtype), gen((B, Hkv, S, D), dtype, 1), gen((B, Hkv, S, D), dtype, 2)
    neg = torch.finfo(dtype).min
    mask = torch.full((B, 1, T, S), neg, dtype=dtype)
    for b in range(B):
        for t in range(T):
            lo = (37 * t + 11 * b) % 300
            mask[b, 0, t, lo:lo + 40 + (t % 64)] = 0          # a sliding window; far tiles are fully masked
        mask[b, 0, :, 128:192] = neg                          # one key tile masked for every row
        mask[b, 0, :, 130 + b] = 0                            # ... except a single key
    mask[1, 0, 150:, 192:256] = torch.where(torch.rand(T - 150, 64, generator=g) < 0.3, 0.0, neg).to(dtype)
    ref = attn_ref(q, k, v, mask, D ** -0.5, dtype).transpose(1, 2)
    Q, K, V, M = q.cuda(), k.cuda(), v.cuda(), mask.cuda()
    out = torch.full((B, T, Hq, D), float("nan"), dtype=dtype, device="cuda")
    st = lambda t: (C.c_int64 * 3)(*t.stride()[:3])
    dt = DT[dtype]
    ok(lib, lib.b200_attn_prefill(Q.data_ptr(), K.data_ptr(), V.data_ptr(), M.data_ptr(), out.data_ptr(), B, Hq, Hkv, T, S, D,
                                  st(Q), st(K), st(V), T * S, S, D ** -0.5, dt, stream()))
    close(out, ref, rtol=2e-2, atol=5e-3)
    ok(lib, lib.b200_attn_prefill(Q.data_ptr(), K.data_ptr(), V.data_ptr(), None, out.data_ptr(), B, Hq, Hkv, T, S, D,
                                  st(Q), st(K), st(V), 0, 0, D ** -0.5, dt, stream()))
    close(out, attn_ref(q, k, v, None, D ** -0.5, dtype).transpose(1, 2), rtol=2e-2, atol=5e-3)
    code = C.c_int(0)
    ok(lib, lib.b200_debug_device_error(C.byref(code), 1))
    assert code.value == 0


# ------------------------------------------------------------------ bandwidth kernels
@pytest.mark.parametrize("rows,cols", [(1, 1536), (128, 1536), (2048, 1536), (5, 4096), (3, 100)])
def test_rmsnorm(lib, rows, cols):
    for dtype in (torch.bfloat16, torch.float16):
        x, w = gen((rows, cols), dtype), (1 + 0.02 * gen((cols,), torch.float32, 1)).to(dtype)
        n = (x.float() * torch.rsqrt(x.float().pow(2).mean(-1, keepdim=True) + 1e-6)).to(dtype)
        ref = (w.float() * n.float()).to(dtype)
        X, W = x.cuda(), w.cuda()
        Y = torch.empty_like(X)
        ok(lib, lib.b200_rmsnorm(X.data_ptr(), W.data_ptr(), Y.data_ptr(), rows, cols, cols, cols, 1e-6, DT[dtype], 1, stream()))
        got, r = Y.cpu(), ref
        ulp = (got.view(torch.int16).int() - r.view(torch.int16).int()).abs()
        # fp32 reduction order only: two roundings, so rarely 2 units in the last place
        assert ulp.max() <= 2 and (ulp != 0).float().mean() < 0.02 and (ulp > 1).float().mean() < 1e-4


@pytest.mark.parametrize("T", [1, 128, 1000, 2048])
def test_masked_softmax(lib, T):
    import model_zoo as mz

    dtype = torch.bfloat16
    H = 12 if T <= 1000 else 3
    x, mask = gen((1, H, T, T), dtype), mz.causal_mask(1, T, T, 0)
    ref = torch.softmax((x.float() + mask.float()).to(dtype).float(), -1)
    X, M = x.cuda(), mask.cuda()
    Y = torch.empty_like(X)
    ok(lib, lib.b200_softmax(X.data_ptr(), M.data_ptr(), Y.data_ptr(), 1, H, T, T, 0, 0, T, 1.0, 2, 2, 2, 1, stream()))
    close(Y, ref, rtol=1e-2, atol=2e-3)
    assert not Y.float().triu(1).any()            # masked positions are exactly zero
    Yf = torch.empty(1, H, T, T, dtype=torch.float32, device="cuda")
    ok(lib, lib.b200_softmax(X.data_ptr(), None, Yf.data_ptr(), 1, H, T, T, 0, 0, 0, 0.5, 2, 0, 0, 0, stream()))
    close(Yf, torch.softmax(x.float() * 0.5, -1), rtol=1e-3, atol=1e-5)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("T", [96, 2048, 8192])
def test_softmax_scale_and_finite_mask_round_like_the_unfused_ops(lib, T, dtype):
    """scale, then an additive mask of arbitrary finite values: each step rounds to the
    input dtype as the separate ATen ops would (the kernel may skip a rounding only where
    it cannot change the value)."""
    H, R = 2, 24
    code = 2 if dtype == torch.bfloat16 else 1
    x, mask = gen((1, H, R, T), dtype), gen((1, 1, R, T), dtype, 1)
    mask[..., ::3] = 0
    mask[..., 1::7] = float("-inf")
    scale = 128 ** -0.5
    ref = torch.softmax(((x.float() * scale).to(dtype).float() + mask.float()).to(dtype).float(), -1)
    X, M = x.cuda(), mask.cuda()
    Y = torch.empty_like(X)
    ok(lib, lib.b200_softmax(X.data_ptr(), M.data_ptr(), Y.data_ptr(), 1, H, R, T, 0, 0, T, scale, code, code, code, 1, stream()))
    close(Y, ref, rtol=1e-2, atol=1e-4)
    if dtype == torch.bfloat16:      # fp16 outputs can sit at the edge of underflow
        assert torch.equal(Y.cpu() == 0, ref.to(dtype) == 0)


def test_softmax_full_size_properties(lib):
    """[12, 8192, 8192] causal: too large for the CPU oracle in a test, so check what must
    hold: rows sum to 1, masked columns are 0, row 0 is one-hot."""
    T, H = 8192, 12
    x = torch.randn(1, H, T, T, device="cuda", dtype=torch.bfloat16, generator=torch.Generator("cuda").manual_seed(0))
    mask = torch.full((T, T), torch.finfo(torch.bfloat16).min, device="cuda", dtype=torch.bfloat16).triu(1)[None, None]
    y = torch.empty_like(x)
    ok(lib, lib.b200_softmax(x.data_ptr(), mask.data_ptr(), y.data_ptr(), 1, H, T, T, 0, 0, T, 1.0, 2, 2, 2, 1, stream()))
    for h in (0, H - 1):
        sums = y[0, h].float().sum(-1)
        assert (sums - 1).abs().max() < 2e-2
        assert not y[0, h].triu(1).any()
        assert y[0, h, 0, 0] == 1


@pytest.mark.parametrize("T", [1, 128, 2048])
def test_silu_mul_and_add_relu_chains(lib, T):
    from cuda_runtime import native

    dtype = torch.bfloat16
    g, u = gen((T, 8960), dtype), gen((T, 8960), dtype, 1)
    G, U = g.cuda(), u.cuda()
    Y = torch.empty_like(G)
    ins = (native.Tensor * 2)(bt(G), bt(U))
    ops = (native.EwOp * 2)(native.EwOp(2, 0, -1, 2, 0.0), native.EwOp(8, 4, 1, 2, 0.0))
    out = bt(Y)
    ok(lib, lib.b200_ew_chain(C.byref(out), ins, 2, ops, 2, stream()))
    ref = (torch.nn.functional.silu(g.float()).to(dtype).float() * u.float()).to(dtype)
    close(Y, ref, rtol=1e-2, atol=1e-2)
    ops = (native.EwOp * 2)(native.EwOp(7, 0, 1, 2, 0.0), native.EwOp(1, 4, -1, 2, 0.0))
    ok(lib, lib.b200_ew_chain(C.byref(out), ins, 2, ops, 2, stream()))
    assert torch.equal(Y.cpu(), torch.relu((g.float() + u.float()).to(dtype)))


def test_ew_chain_broadcast_and_strided(lib):
    from cuda_runtime import native

    x = gen((2, 5, 7, 16), torch.float16).cuda()
    b = gen((1, 5, 1, 1), torch.float32, 1).cuda()
    xt = x.permute(0, 2, 3, 1)                                  # channels-last style view
    y = torch.empty(2, 7, 16, 5, dtype=torch.float16, device="cuda")
    ins = (native.Tensor * 2)(bt(xt), bt(b.permute(0, 2, 3, 1).expand(2, 7, 16, 5)))
    ops = (native.EwOp * 3)(native.EwOp(8, 0, 1, 0, 0.0), native.EwOp(11, 4, -1, 0, 0.25), native.EwOp(3, 5, -1, 1, 0.0))
    out = bt(y)
    ok(lib, lib.b200_ew_chain(C.byref(out), ins, 2, ops, 3, stream()))
    ref = -(xt.float() * b.permute(0, 2, 3, 1) + 0.25)
    close(y, ref, rtol=2e-3, atol=2e-3)


@pytest.mark.parametrize("T", [1, 128, 2048])
def test_rope_table_and_rotate(lib, T):
    dtype, H, D = torch.bfloat16, 12, 128
    inv = 1.0 / (1e6 ** (torch.arange(0, D, 2).float() / D))
    pos = torch.arange(T) + 4096
    ang = torch.cat([pos.float()[:, None] * inv[None]] * 2, -1)
    cos, sin = ang.cos().to(dtype), ang.sin().to(dtype)
    INV, POS = inv.cuda(), pos.cuda()
    Cd, Sd = torch.empty(T, D, dtype=dtype, device="cuda"), torch.empty(T, D, dtype=dtype, device="cuda")
    ok(lib, lib.b200_rope_table(INV.data_ptr(), POS.data_ptr(), Cd.data_ptr(), Sd.data_ptr(), T, D, 4, 2, stream()))
    for got, ref in ((Cd, cos), (Sd, sin)):
        ulp = (got.cpu().view(torch.int16).int() - ref.view(torch.int16).int()).abs()
        assert ulp.max() <= 1 and (ulp != 0).float().mean() < 0.01
    x = gen((1, T, H, D), dtype).transpose(1, 2)
    xf = x.float()
    rot = torch.cat([-xf[..., D // 2:], xf[..., : D // 2]], -1)
    ref = ((xf * cos.float()).to(dtype).float() + (rot * sin.float()).to(dtype).float()).to(dtype)
    X = x.transpose(1, 2).contiguous().cuda().transpose(1, 2)
    Y = torch.empty(1, H, T, D, dtype=dtype, device="cuda")
    xs = bt(X)
    cos_d, sin_d = cos.cuda(), sin.cuda()
    ok(lib, lib.b200_rope_rotate(C.byref(xs), cos_d.data_ptr(), sin_d.data_ptr(), Y.data_ptr(), None, None, 0, 0, stream()))
    assert torch.equal(Y.cpu(), ref)


@pytest.mark.parametrize("M,N,K,fused", [(512, 1536, 8960, True), (1000, 1200, 4104, True), (300, 1536, 1024, False), (64, 1536, 8960, False)])
def test_linear_rmsnorm_equals_the_two_kernels(lib, M, N, K, fused):
    """b200_linear_rmsnorm = b200_linear then b200_rmsnorm.  On the CTA-pair split-K shapes the reduce kernel normalises the
    rows itself (the sum of squares is added in another order: last-bit differences); elsewhere the two kernels run as they are."""
    dtype = torch.bfloat16
    a, w, r = gen((M, K), dtype).cuda(), gen((N, K), dtype, 1, 0.05).cuda(), gen((M, N), dtype, 2).cuda()
    b, g = gen((N,), dtype, 3).cuda(), (1 + 0.1 * gen((N,), dtype, 4).float()).to(dtype).cuda()
    nb = lib.b200_linear_workspace_bytes(M, N, K)
    assert nb > 0 or not fused
    ws = torch.zeros(max(nb, 32), dtype=torch.uint8, device="cuda")
    h1, n1, h2, n2 = (torch.empty(M, N, dtype=dtype, device="cuda") for _ in range(4))
    for round_mid in (1, 0):
        ok(lib, lib.b200_linear_rmsnorm(a.data_ptr(), w.data_ptr(), b.data_ptr(), r.data_ptr(), h1.data_ptr(), M, N, K, K, K, N, N, 2, 2, 0,
                                        ws.data_ptr(), ws.numel(), g.data_ptr(), n1.data_ptr(), N, 1e-6, round_mid, stream()))
        ok(lib, lib.b200_linear(a.data_ptr(), w.data_ptr(), b.data_ptr(), r.data_ptr(), h2.data_ptr(), M, N, K, K, K, N, N, 2, 2, 0, None, 0,
                                ws.data_ptr(), ws.numel(), stream()))
        ok(lib, lib.b200_rmsnorm(h2.data_ptr(), g.data_ptr(), n2.data_ptr(), M, N, N, N, 1e-6, 2, round_mid, stream()))
        torch.cuda.synchronize()
        assert torch.equal(h1, h2)
        assert int(ws.count_nonzero()) == 0                     # the split-K workspace is left zeroed
        if fused:
            ulp = (n1.view(torch.int16).int() - n2.view(torch.int16).int()).abs()
            assert int(ulp.max()) <= 1 and float((ulp != 0).float().mean()) < 0.01
        else:
            assert torch.equal(n1, n2)
        hf = h2.float()
        x = hf * torch.rsqrt(hf.pow(2).mean(-1, keepdim=True) + 1e-6)
        if round_mid:
            x = x.to(dtype).float()
        close(n1, (x * g.float()).cpu(), rtol=2e-2, atol=2e-2)


@pytest.mark.parametrize("B,T", [(1, 512), (2, 37), (1, 5000)])
def test_rope_rotate_pair_equals_two_rotations(lib, B, T):
    """rope(q) and rope(k) of a prefill layer in one call, from column slices of the merged projection's
    output: bit-identical to two b200_rope_rotate calls (5000 positions: the two-launch form inside)."""
    dtype, Hq, Hkv, D = torch.bfloat16, 12, 2, 128
    N = (Hq + 2 * Hkv) * D
    qkv = gen((B, T, N), dtype).cuda()
    inv = 1.0 / (1e6 ** (torch.arange(0, D, 2).float() / D))
    ang = torch.cat([(torch.arange(T) + 3).float()[:, None] * inv[None]] * 2, -1)
    cos = ang.cos().to(dtype)[None].expand(B, T, D).contiguous().cuda()
    sin = ang.sin().to(dtype)[None].expand(B, T, D).contiguous().cuda()
    q = qkv[..., :Hq * D].view(B, T, Hq, D).transpose(1, 2)
    k = qkv[..., Hq * D:(Hq + Hkv) * D].view(B, T, Hkv, D).transpose(1, 2)
    qo, ko = torch.empty(B, Hq, T, D, dtype=dtype, device="cuda"), torch.empty(B, Hkv, T, D, dtype=dtype, device="cuda")
    qr, kr = torch.empty_like(qo), torch.empty_like(ko)
    qs, ks = bt(q), bt(k)
    ok(lib, lib.b200_rope_rotate_pair(C.byref(qs), C.byref(ks), cos.data_ptr(), sin.data_ptr(), qo.data_ptr(), ko.data_ptr(), stream()))
    ok(lib, lib.b200_rope_rotate(C.byref(qs), cos.data_ptr(), sin.data_ptr(), qr.data_ptr(), None, None, 0, 0, stream()))
    ok(lib, lib.b200_rope_rotate(C.byref(ks), cos.data_ptr(), sin.data_ptr(), kr.data_ptr(), None, None, 0, 0, stream()))
    assert torch.equal(qo, qr) and torch.equal(ko, kr)
    xf = k.float().cpu()
    rot = torch.cat([-xf[..., D // 2:], xf[..., : D // 2]], -1)
    c, s_ = cos.cpu().float()[:, None], sin.cpu().float()[:, None]
    assert torch.equal(ko.cpu(), ((xf * c).to(dtype).float() + (rot * s_).to(dtype).float()).to(dtype))
    # mismatched positions are refused
    k_bad = bt(k[:, :, : T - 1])
    assert lib.b200_rope_rotate_pair(C.byref(qs), C.byref(k_bad), cos.data_ptr(), sin.data_ptr(), qo.data_ptr(), ko.data_ptr(), stream()) == -1   # B200_EINVAL


@pytest.mark.parametrize("B,T", [(1, 1), (8, 1), (2, 5)])
def test_qkv_rope_cache_fused(lib, B, T):
    """rope(q), rope(k) -> key cache row, v -> value cache row in one launch, from column
    slices of one merged projection buffer (the layout the compiler produces)."""
    dtype, Hq, Hkv, D, S = torch.bfloat16, 12, 2, 128, 64
    N = (Hq + 2 * Hkv) * D
    qkv = gen((B, T, N), dtype)
    pos = torch.arange(T) + 17
    inv = 1.0 / (1e6 ** (torch.arange(0, D, 2).float() / D))
    ang = torch.cat([pos.float()[:, None] * inv[None]] * 2, -1)
    cos = ang.cos().to(dtype)[None].expand(B, T, D).contiguous()
    sin = ang.sin().to(dtype)[None].expand(B, T, D).contiguous()
    kc, vc = gen((B, Hkv, S, D), dtype, 1), gen((B, Hkv, S, D), dtype, 2)

    def heads(lo, n):  # [B,T,n*D] column slice -> [B,n,T,D] view
        return qkv[..., lo:lo + n * D].view(B, T, n, D).transpose(1, 2)

    def rope(x):
        xf = x.float()
        rot = torch.cat([-xf[..., D // 2:], xf[..., : D // 2]], -1)
        return ((xf * cos[:, None].float()).to(dtype).float() + (rot * sin[:, None].float()).to(dtype).float()).to(dtype)

    q, k, v = heads(0, Hq), heads(Hq * D, Hkv), heads((Hq + Hkv) * D, Hkv)
    ref_q = rope(q)
    ref_k, ref_v = kc.clone(), vc.clone()
    ref_k[:, :, pos] = rope(k)
    ref_v[:, :, pos] = v
    QKV, KC, VC, CO, SI, P = qkv.cuda(), kc.cuda(), vc.cuda(), cos.cuda(), sin.cuda(), pos.cuda()
    dv = lambda lo, n: QKV[..., lo:lo + n * D].view(B, T, n, D).transpose(1, 2)
    tq, tk, tv = bt(dv(0, Hq)), bt(dv(Hq * D, Hkv)), bt(dv((Hq + Hkv) * D, Hkv))
    qo = torch.empty(B, Hq, T, D, dtype=dtype, device="cuda")
    ok(lib, lib.b200_qkv_rope_cache(C.byref(tq), C.byref(tk), C.byref(tv), CO.data_ptr(), SI.data_ptr(), qo.data_ptr(), KC.data_ptr(),
                                    VC.data_ptr(), P.data_ptr(), S, 4, stream()))
    assert torch.equal(qo.cpu(), ref_q) and torch.equal(KC.cpu(), ref_k) and torch.equal(VC.cpu(), ref_v)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("B,norm,pos", [(1, True, 17), (8, True, 4100), (64, True, 4351), (5, False, -3), (64, False, 0), (9, True, 0),
                                        (16, True, 4351), (17, False, 5), (19, True, 613), (24, True, -1), (25, True, 3)])
def test_linear_qkv_rope_equals_the_two_kernels(lib, dtype, B, norm, pos):
    """The merged q/k/v projection whose final pass rotates q and k and writes the cache rows is
    bit-identical to the projection followed by the rope / cache kernel - q, both caches whole."""
    Hq, Hkv, D, S, K = 12, 2, 128, 4352, 1536
    N = (Hq + 2 * Hkv) * D
    DTC = DT[dtype]
    x = gen((B, K), dtype, 0, 2.0).cuda()
    w, bias = gen((N, K), dtype, 1, 0.03).cuda(), gen((N,), dtype, 2).cuda()
    sumsq = x.float().pow(2).reshape(B, 24, K // 24).sum(-1).contiguous() if norm else None
    p_abs = pos if pos >= 0 else S + pos
    inv = 1.0 / (1e6 ** (torch.arange(0, D, 2).float() / D))
    ang = torch.cat([torch.full((B, 1), float(p_abs)) * inv[None]] * 2, -1)
    CO, SI = ang.cos().to(dtype).cuda().contiguous(), ang.sin().to(dtype).cuda().contiguous()
    kc0, vc0 = gen((B, Hkv, S, D), dtype, 3).cuda(), gen((B, Hkv, S, D), dtype, 4).cuda()
    P = torch.tensor([pos], dtype=torch.int64, device="cuda")
    sq_ptr, n_part = (sumsq.data_ptr(), 24) if norm else (None, 0)
    # two kernels
    qkv = torch.empty(B, N, dtype=dtype, device="cuda")
    ok(lib, lib.b200_linear_norm(x.data_ptr(), w.data_ptr(), bias.data_ptr(), None, qkv.data_ptr(), B, N, K, K, K, N, 0, DTC, DTC, 8,
                                 1e-6, sq_ptr, n_part, None, stream()))
    dv = lambda lo, n: qkv[:, None, lo:lo + n * D].view(B, 1, n, D).transpose(1, 2)
    tq, tk, tv = bt(dv(0, Hq)), bt(dv(Hq * D, Hkv)), bt(dv((Hq + Hkv) * D, Hkv))
    q_ref, k_ref, v_ref = torch.empty(B, Hq, 1, D, dtype=dtype, device="cuda"), kc0.clone(), vc0.clone()
    ok(lib, lib.b200_qkv_rope_cache(C.byref(tq), C.byref(tk), C.byref(tv), CO.data_ptr(), SI.data_ptr(), q_ref.data_ptr(), k_ref.data_ptr(),
                                    v_ref.data_ptr(), P.data_ptr(), S, 4, stream()))
    # one kernel
    q_out, kc, vc = torch.full((B, Hq, 1, D), float("nan"), dtype=dtype, device="cuda"), kc0.clone(), vc0.clone()
    ok(lib, lib.b200_linear_qkv_rope(x.data_ptr(), w.data_ptr(), bias.data_ptr(), B, N, K, K, K, DTC, DTC, 8, 1e-6, sq_ptr, n_part,
                                     CO.data_ptr(), SI.data_ptr(), q_out.data_ptr(), kc.data_ptr(), vc.data_ptr(), P.data_ptr(), S, 4, Hq, Hkv,
                                     stream()))
    torch.cuda.synchronize()
    as_bits = lambda t: t.cpu().view(torch.int16)
    assert torch.equal(as_bits(q_out), as_bits(q_ref))
    assert torch.equal(as_bits(kc), as_bits(k_ref)) and torch.equal(as_bits(vc), as_bits(v_ref))
    assert not torch.equal(as_bits(kc[:, :, p_abs]), as_bits(kc0[:, :, p_abs]))       # the row was written
    code = C.c_int(-1)
    ok(lib, lib.b200_debug_device_error(C.byref(code), 1))
    assert code.value == 0


def test_linear_qkv_rope_rejects_what_it_cannot_fuse(lib):
    x, w = gen((65, 1536), torch.bfloat16).cuda(), gen((2048, 1536), torch.bfloat16, 1).cuda()
    t = torch.zeros(65 * 12 * 128, dtype=torch.bfloat16, device="cuda")
    P = torch.zeros(1, dtype=torch.int64, device="cuda")
    args = lambda M, N, Hq: (x.data_ptr(), w.data_ptr(), None, M, N, 1536, 1536, 1536, 2, 2, 8, 0.0, None, 0, t.data_ptr(), t.data_ptr(),
                             t.data_ptr(), t.data_ptr(), t.data_ptr(), P.data_ptr(), 16, 4, Hq, 2, stream())
    assert lib.b200_linear_qkv_rope(*args(65, 2048, 12)) == -4      # more than 64 rows: B200_ENOTSUP
    assert lib.b200_linear_qkv_rope(*args(8, 2048, 10)) == -1       # N != (Hq + 2 Hkv) * 128: B200_EINVAL


def test_embedding_is_bit_exact(lib):
    V, D = 151936, 1536
    table = torch.randn(V, D, generator=torch.Generator().manual_seed(0)).bfloat16()
    ids = torch.tensor([0, V - 1, 70000, 65505, 2049, 151935, 1, 1], dtype=torch.int64)
    Tb, I = table.cuda(), ids.cuda()
    out = torch.empty(len(ids), D, dtype=torch.bfloat16, device="cuda")
    ok(lib, lib.b200_embedding(Tb.data_ptr(), I.data_ptr(), out.data_ptr(), len(ids), V, D * 2, 4, stream()))
    assert torch.equal(out.cpu().view(torch.int16), table[ids].view(torch.int16))
    I32 = ids.int().cuda()
    ok(lib, lib.b200_embedding(Tb.data_ptr(), I32.data_ptr(), out.data_ptr(), len(ids), V, D * 2, 3, stream()))
    assert torch.equal(out.cpu().view(torch.int16), table[ids].view(torch.int16))
    ok(lib, lib.b200_embedding(Tb.data_ptr(), I.data_ptr(), out.data_ptr(), 0, V, D * 2, 4, stream()))  # empty gather


@pytest.mark.parametrize("in_place", [True, False])
def test_index_copy_is_bit_exact(lib, in_place):
    B, H, S, D = 3, 2, 4352, 128
    cache, src = gen((B, H, S, D)), gen((B, 1, H, D), seed=1).transpose(1, 2)   # src is a strided view, as in the graph
    pos = torch.tensor([4100])
    ref = cache.index_copy(2, pos, src)
    Cc, Sc, P = cache.cuda(), src.transpose(1, 2).contiguous().cuda().transpose(1, 2), pos.cuda()
    dst = Cc if in_place else torch.zeros_like(Cc)
    ok(lib, lib.b200_index_copy(Cc.data_ptr(), dst.data_ptr(), Sc.data_ptr(), P.data_ptr(), B * H, S, D, 1, D, D * H, 2, 4, stream()))
    assert torch.equal(dst.cpu().view(torch.int16), ref.view(torch.int16))


def test_strided_copy_transpose_cast_and_pad(lib):
    x = gen((2, 3, 20, 20), torch.float32)
    X = x.cuda()
    full = torch.zeros(2, 20, 20, 8, dtype=torch.float16, device="cuda")
    dst = full.permute(0, 3, 1, 2)[:, :3]                       # NCHW-shaped window of an NHWC8 buffer
    a, b = bt(dst), bt(X)
    ok(lib, lib.b200_strided_copy(C.byref(a), C.byref(b), stream()))
    assert torch.equal(full[..., :3].cpu(), x.permute(0, 2, 3, 1).half()) and not full[..., 3:].any()
    y = gen((4, 6, 128), torch.bfloat16).cuda()
    z = torch.empty(6, 4, 128, dtype=torch.bfloat16, device="cuda")
    a, b = bt(z), bt(y.transpose(0, 1))
    ok(lib, lib.b200_strided_copy(C.byref(a), C.byref(b), stream()))
    assert torch.equal(z, y.transpose(0, 1).contiguous())


@pytest.mark.parametrize("N,Cn,H,W", [(3, 3, 5, 7), (2, 8, 4, 6), (1, 2, 33, 31)])
def test_strided_copy_planar_to_eight_channel_slots(lib, N, Cn, H, W):
    """Same-dtype NCHW -> NHWC8 window (the input repack of a convolution network): the
    channels of the window are replaced, the other channels of each slot keep their contents."""
    x = gen((N, Cn, H, W), torch.float16)
    X = x.cuda()
    full = torch.full((N, H, W, 8), 7.0, dtype=torch.float16, device="cuda")
    dst = full.permute(0, 3, 1, 2)[:, :Cn]
    a, b = bt(dst), bt(X)
    ok(lib, lib.b200_strided_copy(C.byref(a), C.byref(b), stream()))
    assert torch.equal(full[..., :Cn].cpu(), x.permute(0, 2, 3, 1))
    assert bool((full[..., Cn:] == 7.0).all())


def test_pooling_and_batchnorm(lib):
    x = gen((2, 64, 112, 112), torch.float16)
    for cl in (True, False):
        X = x.cuda().contiguous(memory_format=torch.channels_last) if cl else x.cuda()
        Y = torch.empty(2, 64, 56, 56, dtype=torch.float16, device="cuda")
        Y = Y.contiguous(memory_format=torch.channels_last) if cl else Y
        a, b = bt(X), bt(Y)
        ok(lib, lib.b200_max_pool2d(C.byref(a), C.byref(b), 3, 3, 2, 2, 1, 1, stream()))
        assert torch.equal(Y.cpu(), torch.nn.functional.max_pool2d(x.float(), 3, 2, 1).half())
        Z = torch.empty(2, 64, 1, 1, dtype=torch.float16, device="cuda")
        c = bt(Z)
        ok(lib, lib.b200_adaptive_avg_pool2d(C.byref(a), C.byref(c), stream()))
        close(Z, x.float().mean((2, 3), keepdim=True), rtol=2e-3, atol=2e-3)
    g, be, m, v = (torch.rand(64) + 0.5).cuda(), torch.randn(64).cuda(), torch.randn(64).cuda(), (torch.rand(64) + 0.5).cuda()
    X = x.cuda()
    Y = torch.empty_like(X)
    a, b = bt(X), bt(Y)
    ok(lib, lib.b200_batch_norm(C.byref(a), C.byref(b), g.data_ptr(), be.data_ptr(), m.data_ptr(), v.data_ptr(), 1e-5, 0, 0, stream()))
    close(Y, torch.nn.functional.batch_norm(x.float(), m.cpu(), v.cpu(), g.cpu(), be.cpu(), False, 0.0, 1e-5), rtol=2e-3, atol=4e-3)


def test_matmul_strided_and_mean_and_fill(lib):
    a, b = gen((2, 3, 20, 24), torch.bfloat16), gen((2, 1, 17, 24), torch.bfloat16, 1)
    A, B = a.cuda(), b.cuda()
    Bt = B.transpose(2, 3).expand(2, 3, 24, 17)
    out = torch.empty(2, 3, 20, 17, dtype=torch.bfloat16, device="cuda")
    arr = lambda t: (C.c_int64 * 4)(*t.stride())
    ok(lib, lib.b200_matmul_strided(A.data_ptr(), Bt.data_ptr(), out.data_ptr(), 2, 3, 20, 17, 24, arr(A), arr(Bt), arr(out), 2, stream()))
    close(out, a.float() @ b.float().transpose(2, 3), rtol=1e-2, atol=5e-2)
    x = gen((50, 333), torch.float32).cuda()
    y = torch.empty(50, dtype=torch.float32, device="cuda")
    ok(lib, lib.b200_mean_last_dim(x.data_ptr(), y.data_ptr(), 50, 333, 0, 0, stream()))
    close(y, x.mean(-1), rtol=1e-5, atol=1e-6)
    z = torch.empty(1000, dtype=torch.bfloat16, device="cuda")
    ok(lib, lib.b200_fill(z.data_ptr(), 1000, -2.5, 2, stream()))
    assert (z == -2.5).all()


def test_argmax_rows_matches_and_breaks_ties_low(lib):
    x = gen((9, 151936), torch.bfloat16)
    x[3, 77] = x[3, 150000] = 50.0
    X = x.cuda()
    out = torch.empty(9, dtype=torch.int64, device="cuda")
    ok(lib, lib.b200_argmax_rows(X.data_ptr(), out.data_ptr(), 9, 151936, 151936, 2, stream()))
    ref = torch.tensor([int(np.flatnonzero(r == r.max())[0]) for r in x.float().numpy()])
    assert torch.equal(out.cpu(), ref) and out[3] == 77


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("N,Cn,H,W,O,KH,ph,relu", [
    (1, 3, 224, 224, 64, 7, 3, True), (5, 3, 224, 224, 64, 7, 3, True),        # one pooled row per CTA; windows that cross images
    (40, 3, 64, 64, 64, 7, 3, True), (7, 3, 65, 71, 48, 7, 3, True),           # several images per CTA; odd sizes, rows that are no whole words
    (3, 4, 32, 256, 8, 7, 3, False), (2, 1, 30, 250, 16, 8, 3, False),         # widest rows, one and four planes, no ReLU, eight filter rows
    (300, 2, 7, 9, 24, 7, 0, True), (4, 3, 1, 8, 64, 3, 1, True), (33, 3, 5, 16, 64, 5, 2, False)])   # images of one or two output rows
def test_conv_stem_pool(lib, dtype, N, Cn, H, W, O, KH, ph, relu):
    """Convolution, bias, ReLU and max-pooling from the planar image in one kernel.  Bound: each convolution output is rounded to the
    activation type once (2^-11 in fp16, 2^-8 in bf16, of its value) after an fp32 sum of at most KH * 28 products (2^-22 of their
    magnitudes); a maximum errs by no more than the largest error under it."""
    x, w = gen((N, Cn, H, W), dtype), gen((O, Cn, KH, 7), dtype, 1, 0.2)
    bias = gen((O,), torch.float32, 2)
    packed = torch.zeros(O, KH, 7, 8, dtype=dtype)
    packed[..., :Cn] = w.permute(0, 2, 3, 1)
    conv = lambda a, b: torch.nn.functional.conv2d(a, b, None, 2, (ph, 3))
    ref, size = conv(x.double(), w.double()) + bias.double()[None, :, None, None], conv(x.double().abs(), w.double().abs()) + bias.double().abs()[None, :, None, None]
    ref = torch.relu(ref) if relu else ref
    pool = lambda t: torch.nn.functional.max_pool2d(t, 3, 2, 1)
    want, slack = pool(ref).permute(0, 2, 3, 1), pool(ref.abs() * (2.0 ** -11 if dtype == torch.float16 else 2.0 ** -8) + size * 2.0 ** -20 + 1e-7).permute(0, 2, 3, 1)
    X, Wd, Bd = x.cuda(), packed.cuda(), bias.cuda()
    y = torch.full(want.shape, float("nan"), dtype=dtype, device="cuda")
    code = DT[dtype]
    assert lib.b200_conv_stem_pool_supported(Cn, H, W, 8, O, KH, 7, 2, 2, ph, 3, code)
    for _ in range(2):
        ok(lib, lib.b200_conv_stem_pool(X.data_ptr(), Wd.data_ptr(), Bd.data_ptr(), y.data_ptr(), N, Cn, H, W, 8, O, KH, 7, 2, 2, ph, 3, code, int(relu), stream()))
    err = (y.double().cpu() - want).abs()
    assert (err <= slack).all(), float((err / slack).max())
    c = C.c_int(0)
    ok(lib, lib.b200_debug_device_error(C.byref(c), 1))
    assert c.value == 0


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("W", [64, 71])
@pytest.mark.parametrize("relu", [True, False])
def test_conv_stem_pool_infinite_pixel(lib, dtype, W, relu):
    """One infinite pixel reaches the outputs whose filter covers it and no other.  Bound of the finite ones as above."""
    x, w = gen((2, 3, 33, W), dtype), gen((64, 3, 7, 7), dtype, 1, 0.2)
    packed = torch.zeros(64, 7, 7, 8, dtype=dtype)
    packed[..., :3] = w.permute(0, 2, 3, 1)
    conv = lambda a, b: torch.nn.functional.conv2d(a, b, None, 2, 3)
    pool = lambda t: torch.nn.functional.max_pool2d(t, 3, 2, 1).permute(0, 2, 3, 1)
    size = conv(x.double().abs(), w.double().abs())
    for at in (0, 12, 13, W - 1):
        bad = x.clone()
        bad[1, 2, 16, at] = float("inf")
        ref = conv(bad.double(), w.double())
        ref = torch.relu(ref) if relu else ref
        want, X, Wd = pool(ref), bad.cuda(), packed.cuda()
        slack = pool(size) * ((2.0 ** -11 if dtype == torch.float16 else 2.0 ** -8) + 2.0 ** -20) + 1e-7
        y = torch.empty(want.shape, dtype=dtype, device="cuda")
        ok(lib, lib.b200_conv_stem_pool(X.data_ptr(), Wd.data_ptr(), None, y.data_ptr(), 2, 3, 33, W, 8, 64, 7, 7, 2, 2, 3, 3, DT[dtype], int(relu), stream()))
        got, finite = y.double().cpu(), want.isfinite()
        assert torch.equal(got[~finite], want[~finite])
        assert got[finite].isfinite().all() and ((got - want).abs()[finite] <= slack[finite]).all()


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_conv_stem_pool_behind_the_kernel_that_prepares_its_weights(lib, dtype):
    """Weights and bias written by the launch before, over and over: each call sees its own, bit for bit."""
    N, H, W, O = 4, 64, 64, 64
    x = gen((N, 3, H, W), dtype).cuda()
    sets = [(gen((O, 3, 7, 7), torch.float32, s, 0.1).cuda(), gen((O,), torch.float32, s + 50).cuda()) for s in range(24)]
    packed, bias = torch.empty(O, 7, 7, 8, dtype=dtype, device="cuda"), torch.empty(O, dtype=torch.float32, device="cuda")
    outs = [torch.full((N, 16, 16, O), float("nan"), dtype=dtype, device="cuda") for _ in range(2 * len(sets))]

    def call(i, out, wait):
        w, b = sets[i]
        go(lib, lib.b200_conv_weight_prep(w.data_ptr(), b.data_ptr(), None, None, None, None, packed.data_ptr(), bias.data_ptr(), O, 3, 7, 7, 8, 0.0, 0, 0, DT[dtype], stream()))
        if wait:
            torch.cuda.synchronize()
        go(lib, lib.b200_conv_stem_pool(x.data_ptr(), packed.data_ptr(), bias.data_ptr(), out.data_ptr(), N, 3, H, W, 8, O, 7, 7, 2, 2, 3, 3, DT[dtype], 1, stream()))

    for i in range(len(sets)):
        call(i, outs[i], False)
    for i in range(len(sets)):
        call(i, outs[len(sets) + i], True)
    for i in range(len(sets)):
        assert torch.equal(outs[i], outs[len(sets) + i]) and outs[i].isfinite().all()
    assert not torch.equal(outs[0], outs[1])


def test_conv_stem_pool_shapes_it_does_not_take(lib):
    for bad in [(5, 32, 32, 8, 64, 7, 7, 2, 2, 3, 3, 1), (3, 32, 258, 8, 64, 7, 7, 2, 2, 3, 3, 1), (3, 32, 32, 8, 72, 7, 7, 2, 2, 3, 3, 1), (3, 32, 32, 8, 64, 9, 7, 2, 2, 3, 3, 1),
                (3, 32, 32, 8, 64, 7, 7, 1, 1, 3, 3, 1), (3, 32, 32, 8, 64, 7, 5, 2, 2, 3, 3, 1), (3, 32, 32, 8, 64, 7, 7, 2, 2, 3, 3, 0)]:
        assert lib.b200_conv_stem_pool_supported(*bad) == 0


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("N,Cn,H,W,OH,OW", [(1, 8, 1, 1, 1, 1), (2, 248, 7, 7, 1, 1), (1, 264, 9, 5, 1, 1), (3, 2048, 7, 7, 1, 1), (2, 64, 13, 11, 4, 3), (2, 20, 7, 7, 1, 1)])
def test_adaptive_avg_pool_channels_last(lib, dtype, N, Cn, H, W, OH, OW):
    """Channels that end inside a block, windows of unequal size, and channels that are no whole words (the general kernel).  One
    rounding of an fp32 mean: 2^-11 in fp16 and 2^-8 in bf16 of the result, 2^-20 of the mean magnitude for the sum."""
    x = gen((N, Cn, H, W), dtype)
    want = torch.nn.functional.adaptive_avg_pool2d(x.double(), (OH, OW))
    size = torch.nn.functional.adaptive_avg_pool2d(x.double().abs(), (OH, OW))
    X = x.cuda().contiguous(memory_format=torch.channels_last)
    Y = torch.full((N, OH, OW, Cn), float("nan"), dtype=dtype, device="cuda").permute(0, 3, 1, 2)
    a, b = bt(X), bt(Y)
    ok(lib, lib.b200_adaptive_avg_pool2d(C.byref(a), C.byref(b), stream()))
    err = (Y.double().cpu() - want).abs()
    assert (err <= want.abs() * (2.0 ** -11 if dtype == torch.float16 else 2.0 ** -8) + size * 2.0 ** -20 + 6e-8).all(), float(err.max())


@pytest.mark.parametrize("N,Cn,H,OH,kernel", [(592, 8, 2, 1, "adaptive_avg_pool2d_cl8_kernel"), (593, 8, 7, 1, "adaptive_avg_pool2d_kernel"), (4000, 64, 11, 1, "adaptive_avg_pool2d_kernel"),
                                              (2000, 64, 13, 1, "adaptive_avg_pool2d_cl8_kernel"), (700, 248, 2, 1, "adaptive_avg_pool2d_cl8_kernel"), (700, 512, 7, 7, "adaptive_avg_pool2d_cl8_kernel"),
                                              (40, 512, 14, 7, "adaptive_avg_pool2d_cl8_kernel"), (700, 264, 6, 1, "adaptive_avg_pool2d_kernel"), (700, 264, 7, 1, "adaptive_avg_pool2d_cl8_kernel")])
def test_adaptive_avg_pool_runs_on_the_kernel_that_its_shape_calls_for(lib, N, Cn, H, OH, kernel):
    """Both sides of each line of the rule (resident blocks, work per block, idle channels), and the result there."""
    x = gen((N, Cn, H, H), torch.float16).cuda().contiguous(memory_format=torch.channels_last)
    y = torch.empty(N, OH, OH, Cn, dtype=torch.float16, device="cuda").permute(0, 3, 1, 2)
    a, b = bt(x), bt(y)
    names = kernels_of(lambda: go(lib, lib.b200_adaptive_avg_pool2d(C.byref(a), C.byref(b), stream())))
    assert len(names) == 1 and kernel in names[0], names
    want = torch.nn.functional.adaptive_avg_pool2d(x.double(), OH)
    size = torch.nn.functional.adaptive_avg_pool2d(x.double().abs(), OH)
    assert ((y.double() - want).abs() <= want.abs() * 2.0 ** -11 + size * 2.0 ** -20 + 6e-8).all()


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("N,H,W,Cn,O,res,relu", [
    (7, 56, 56, 64, 64, False, True), (12, 56, 56, 64, 64, True, True),      # weights resident, two issuing threads; with residual
    (20, 31, 30, 64, 64, False, False), (9, 57, 55, 64, 40, True, False),    # last tiles of an image shorter, fewer channels than a tile
    (3, 90, 126, 64, 64, False, True), (25, 28, 28, 128, 128, True, True),   # one row per tile; weights streamed, one tile per unit
    (127, 28, 28, 128, 128, False, True), (20, 28, 28, 64, 200, True, True),  # one tile per unit; two, and two column tiles
    (125, 28, 28, 128, 128, False, True), (125, 28, 28, 128, 128, True, False),   # two tiles per unit, an odd number of tiles
    (21, 28, 28, 64, 200, True, True), (41, 28, 28, 64, 200, False, False),      # the same in each of two column tiles
    (35, 14, 14, 256, 256, True, True), (40, 14, 14, 192, 136, False, True), (300, 7, 15, 64, 128, False, True),   # tiles of eight rows; a whole image per tile
    (48, 14, 14, 256, 256, True, True)])                                     # (the im2col route)
def test_conv3x3_rows(lib, dtype, N, H, W, Cn, O, res, relu):
    """3x3 / 1 / 1 convolutions over enough pixels for the kernel that keeps input rows in shared memory.  Bound: fp32 sums of 9 C
    products (2^-20 of their magnitudes), rounded to the activation type, the sum with the residual rounded once more."""
    x, w = gen((N, H, W, Cn), dtype).cuda(), gen((O, 3, 3, Cn), dtype, 1, 0.05).cuda()
    bias = gen((O,), torch.float32, 2).cuda()
    r = gen((N, H, W, O), dtype, 3).cuda() if res else None
    conv = lambda a, b: torch.nn.functional.conv2d(a.permute(0, 3, 1, 2), b.permute(0, 3, 1, 2), None, 1, 1).permute(0, 2, 3, 1)
    eps = 2.0 ** -11 if dtype == torch.float16 else 2.0 ** -8
    want = conv(x.double(), w.double()) + bias.double()
    slack = want.abs() * eps + (conv(x.double().abs(), w.double().abs()) + bias.double().abs()) * 2.0 ** -20 + 1e-7
    if res:
        want = want + r.double()
        slack = slack + want.abs() * eps
    want = torch.relu(want) if relu else want
    y = torch.full((N, H, W, O), float("nan"), dtype=dtype, device="cuda")
    for _ in range(2):
        ok(lib, lib.b200_conv2d_nhwc(x.data_ptr(), w.data_ptr(), bias.data_ptr(), r.data_ptr() if res else None, y.data_ptr(), N, H, W, Cn, Cn, O, 3, 3, 1, 1, 1, 1,
                                     H, W, DT[dtype], int(relu), stream()))
        err = (y.double() - want).abs()
        assert (err <= slack * 1.01).all(), float((err / slack).max())
    code = C.c_int(0)
    ok(lib, lib.b200_debug_device_error(C.byref(code), 1))
    assert code.value == 0


@pytest.mark.parametrize("N,H,Cn,O,kernel", [(20, 56, 64, 64, "conv_rows_kernel<__half, 64, 1, true>"), (127, 28, 128, 128, "conv_rows_kernel<__half, 128, 1, false>"),
                                             (20, 28, 128, 128, "conv_rows_kernel<__half, 128, 1, false>"), (125, 28, 128, 128, "conv_rows_kernel<__half, 128, 2, false>"),
                                             (20, 28, 64, 200, "conv_rows_kernel<__half, 128, 2, false>"), (21, 28, 64, 200, "conv_rows_kernel<__half, 128, 2, false>"),
                                             (48, 14, 256, 256, "gemm_tc5p_kernel"), (256, 14, 256, 256, "gemm_tc5p_kernel"), (20, 56, 128, 64, "gemm_tc5p_kernel"),
                                             (2, 56, 64, 64, "gemm_tc5_kernel")])
def test_conv3x3_runs_on_the_kernel_that_its_shape_calls_for(lib, N, H, Cn, O, kernel):
    x, w = torch.zeros(N, H, H, Cn, dtype=torch.float16, device="cuda"), torch.zeros(O, 3, 3, Cn, dtype=torch.float16, device="cuda")
    y = torch.empty(N, H, H, O, dtype=torch.float16, device="cuda")
    call = lambda: go(lib, lib.b200_conv2d_nhwc(x.data_ptr(), w.data_ptr(), None, None, y.data_ptr(), N, H, H, Cn, Cn, O, 3, 3, 1, 1, 1, 1, H, H, 1, 0, stream()))
    names = kernels_of(call)
    assert len(names) == 1 and kernel in names[0], names


@pytest.mark.parametrize("M,form", [(M, form) for M in (65, 80, 128, 129, 250, 257, 273, 500, 777) for form in (
    "plain", "plain odd", "residual", "residual relu", "residual unaligned", "gated", "gated unaligned", "silu mul", "silu mul aligned", "split") if form != "split" or M > 256])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_linear_pair_token_tiles(lib, M, form, dtype):
    """Token tiles of every width (multiples of 16, a last one that is short), each epilogue, partial sums; columns that end inside a
    block; rows that are whole 16-byte words and rows that are not.  Bound: fp32 sums of K products (2^-20 of their magnitudes), each
    rounding to the activation type 2^-8 (bf16) or 2^-11."""
    N, K = (9600, 1032) if form != "split" else (1536, 4104)
    if form in ("residual unaligned", "silu mul"):
        N = 9500
    if form == "plain odd":
        N = 9501
    a, w, bias = gen((M, K), dtype).cuda(), gen((N, K), dtype, 1, 0.05).cuda(), gen((N,), torch.float32, 2).cuda()
    eps = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    s, size = a.double() @ w.double().T + bias.double(), a.double().abs() @ w.double().abs().T + bias.double().abs()
    slack = s.abs() * eps + size * 2.0 ** -20 + 1e-6
    epi, res, aux, out_cols = 0, None, None, N
    if form in ("gated", "gated unaligned"):
        epi, out_cols = 4, N // 2
        blocks, sb = s.view(M, N // 128, 2, 64), slack.view(M, N // 128, 2, 64)
        gate, up = blocks[:, :, 0], blocks[:, :, 1]
        act = gate * torch.sigmoid(gate)
        want = (act * up).reshape(M, -1)
        slack = ((sb[:, :, 0] * 1.1 + act.abs() * (eps + 1e-5)) * up.abs() + act.abs() * sb[:, :, 1] + 2 * sb[:, :, 0] * sb[:, :, 1]).reshape(M, -1) + want.abs() * eps + 1e-6
    elif form in ("silu mul", "silu mul aligned"):
        epi, aux = 2, gen((M, N), dtype, 3).cuda()
        act = s * torch.sigmoid(s)
        want = act * aux.double()
        slack = (slack * 1.1 + act.abs() * (eps + 1e-5)) * aux.double().abs() + want.abs() * eps + 1e-6
    elif form in ("plain", "plain odd"):
        want = s
    else:
        res = gen((M, N), dtype, 3).cuda()
        want = s + res.double()
        slack = slack + want.abs() * eps
        if form == "residual relu":
            epi, want = 1, torch.relu(want)
    ldo = out_cols + (3 if form == "gated unaligned" else 0)
    rows = torch.full((M, ldo), float("nan"), dtype=dtype, device="cuda")
    out = rows[:, :out_cols]
    need = lib.b200_linear_workspace_bytes(M, N, K)
    assert (need > 0) == (form == "split")
    ws = torch.zeros(max(need, 16), dtype=torch.uint8, device="cuda")
    for _ in range(2):
        ok(lib, lib.b200_linear(a.data_ptr(), w.data_ptr(), bias.data_ptr(), res.data_ptr() if res is not None else None, out.data_ptr(), M, N, K, K, K, ldo,
                                N if res is not None else 0, DT[dtype], 0, epi, aux.data_ptr() if aux is not None else None, N if aux is not None else 0,
                                ws.data_ptr(), need, stream()))
        err = (out.double() - want).abs()
        assert (err <= slack * 1.01).all(), float((err / slack).max())
    assert rows[:, out_cols:].isnan().all()
    code = C.c_int(0)
    ok(lib, lib.b200_debug_device_error(C.byref(code), 1))
    assert code.value == 0
