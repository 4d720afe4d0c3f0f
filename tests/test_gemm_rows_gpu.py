"""Products of few rows (gemm_rows.cu, skinny_linear.cu) against float64: every padding of the batch, ragged widths and depths, tiles shared
by several blocks, one block over several tiles, packed weights, the epilogue, and the same bits from run to run."""
import pytest
import torch

from transformers_fusion_b200.ops import _lib, functional as F
from transformers_fusion_b200.quant import wq

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return ((a.double() - b).norm() / b.norm()).item()


def _rows(x, w, out, bias=None, residual=None, alpha=1.0, act=0):
    _lib.check(_lib.lib().tfb_gemm_rows(x.data_ptr(), x.stride(0), w.data_ptr(), w.stride(0), out.data_ptr(), out.stride(0), x.shape[0], w.shape[0],
                                        x.shape[1], _lib.ptr(bias), _lib.ptr(residual), residual.stride(0) if residual is not None else 0, alpha, act,
                                        int(out.dtype == torch.float32), 0, _lib.status_word().data_ptr(), _lib.stream()), "gemm_rows")


# 128 x 64: one unit; 40 x 8: less than a tile and a k-block; 4096 x 14336: five blocks share a tile; 20000 x 200: a block holds several tiles
@pytest.mark.parametrize("N,K", [(128, 64), (40, 8), (1536, 512), (1000, 776), (6144, 4096), (4096, 14336), (20000, 200)])
@pytest.mark.parametrize("M", [1, 16, 17, 33, 64, 65, 128])
def test_gemm_rows(M, N, K):
    g = torch.Generator(device="cuda").manual_seed(M * 7 + N)
    x = torch.randn(M, K, device="cuda", generator=g).bfloat16()
    w = (torch.randn(N, K, device="cuda", generator=g) * K ** -0.5).bfloat16()
    ref = x.double() @ w.double().t()
    outs = []
    for _ in range(3):          # counters and partial sums are left ready for the next product
        out = torch.full((M, N), float("nan"), device="cuda", dtype=torch.float32)
        _rows(x, w, out)
        outs.append(out)
    torch.cuda.synchronize()
    _lib.check_status()
    # fp32 sums of K products of bf16 values: rounding errors of about sqrt(K) 2^-24
    assert _rel(outs[0], ref) < 2e-6 + 1e-7 * K ** 0.5
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])


@pytest.mark.parametrize("M,N,K", [(3, 1000, 4096), (16, 512, 512), (40, 6144, 4096), (64, 1408, 512), (100, 17000, 768)])
def test_few_rows_epilogue(M, N, K):
    """Through the public products: bias, residual with a row pitch of its own, alpha, activation, bf16 and fp32 results, weights fetched ahead."""
    x, w = torch.randn(M, K, device="cuda").bfloat16(), (torch.randn(N, K, device="cuda") * K ** -0.5).bfloat16()
    bias, res = torch.randn(N, device="cuda").bfloat16(), torch.randn(M, N + 24, device="cuda").bfloat16()[:, 8:8 + N]
    prod = x.double() @ w.double().t()
    want = 0.5 * prod + bias.double()
    assert _rel(F.gemm(x, w, bias=bias, residual=res, alpha=0.5), want + res.double()) < 3e-3          # bf16 results: 2^-9
    assert _rel(F.gemm(x, w, bias=bias, alpha=0.5, act="silu"), torch.nn.functional.silu(want)) < 3e-3
    assert _rel(F.gemm(x, w, out_dtype=torch.float32), prod) < 1e-5
    assert _rel(F.linear(x, w, bias, res), prod + bias.double() + res.double()) < 3e-3
    y = torch.empty(M, N + 1, device="cuda", dtype=torch.bfloat16)[:, 1:]                              # rows on odd addresses
    assert _rel(F.gemm(x, w, out=y), prod) < 3e-3
    torch.cuda.synchronize()
    _lib.check_status()


@pytest.mark.parametrize("fmt,group", [("int8", 32), ("int8", 64), ("mxfp8", 32), ("int4", 32), ("fp4", 32), ("ternary", 64)])
@pytest.mark.parametrize("M,N,K", [(1, 128, 64), (5, 1000, 776), (16, 4096, 4096), (9, 28672, 512), (16, 512, 14336), (17, 1536, 512),
                                   (32, 512, 14336)])
def test_packed_rows(M, N, K, fmt, group):
    x, w = torch.randn(M, K, device="cuda").bfloat16(), (torch.randn(N, K, device="cuda") * K ** -0.5).bfloat16()
    bias, res = torch.randn(N, device="cuda").bfloat16(), torch.randn(M, N, device="cuda").bfloat16()
    pw = wq.pack_weight(w, fmt, group)
    # the oracle multiplies unrounded code * scale; the kernel's weights are that in bf16, 2^-9 each
    want = x.double() @ wq.dequant(pw).double().t() + bias.double() + res.double()
    a = wq.gemm_wq(x, pw, bias, residual=res)
    b = wq.gemm_wq(x, pw, bias, residual=res, w_static=True)
    out = torch.empty(M, N, device="cuda", dtype=torch.bfloat16)
    c = wq.gemm_wq(x, pw, bias, residual=res, out=out)
    torch.cuda.synchronize()
    _lib.check_status()
    assert _rel(a, want) < 6e-3 and torch.equal(a, b) and torch.equal(a, c) and c is out


@pytest.mark.parametrize("M", [1, 8, 20])
def test_packed_rows_operands_of_other_layouts(M):
    """What the general form copies or refuses, the one-launch forms do as well: destinations of a wrong shape, on the host, of another
    type or pitch; biases with a stride or on the host; residuals that broadcast."""
    N, K = 520, 256
    x, w = torch.randn(M, K, device="cuda").bfloat16(), (torch.randn(N, K, device="cuda") / 16).bfloat16()
    pw = wq.pack_weight(w, "int8", 32)
    bias = torch.randn(2 * N, device="cuda").bfloat16()[::2]
    want = wq.gemm_wq(x, pw, bias.contiguous())
    for b in (bias, bias.cpu()):
        assert _rel(wq.gemm_wq(x, pw, b), want.double()) < 3e-3
    wide = torch.zeros(M, N + 8, device="cuda", dtype=torch.bfloat16)
    for out in (torch.empty(M, N, dtype=torch.bfloat16), torch.empty(M, N, device="cuda"), wide[:, 8:], torch.empty(N, M, device="cuda", dtype=torch.bfloat16).t()):
        y = wq.gemm_wq(x, pw, bias.contiguous(), out=out)
        assert y is out and _rel(y.cuda(), want.double()) < 3e-3
    assert (wide[:, :8] == 0).all()
    for shape in ((M, N - 8), (M, N + 8), (2, M, N - 1)) + (((M + 1, N),) if M > 1 else ()):      # one row spreads over several
        with pytest.raises(RuntimeError):
            wq.gemm_wq(x, pw, out=torch.empty(shape, device="cuda", dtype=torch.bfloat16))
    res = torch.randn(1, N, device="cuda").bfloat16()
    assert _rel(wq.gemm_wq(x, pw, residual=res), wq.gemm_wq(x, pw).double() + res.double()) < 3e-3
    with pytest.raises(RuntimeError):
        wq.gemm_wq(x, pw, residual=res[:, :-8])
    torch.cuda.synchronize()
    _lib.check_status()


def test_rows_under_capture_and_on_streams():
    """Captured and eager products of one stream give the same bits, and those of many streams the same values."""
    x, w = torch.randn(8, 4096, device="cuda").bfloat16(), (torch.randn(6144, 4096, device="cuda") / 64).bfloat16()
    ref = F.gemm(x, w)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        y = F.linear(F.linear(x, w)[:, :4096].contiguous(), w)
    for _ in range(3):
        graph.replay()
    z = F.linear(ref[:, :4096].contiguous(), w)
    assert torch.equal(y, z)
    outs = []
    torch.cuda.synchronize()
    for _ in range(9):
        s = torch.cuda.Stream()
        with torch.cuda.stream(s):
            outs.append(F.gemm(x, w))
    torch.cuda.synchronize()
    for o in outs:
        assert _rel(o, ref.double()) < 3e-3


def _used(what):
    _lib.register("tfb_rows_workspaces", [_lib.c_i])
    return _lib.lib().tfb_rows_workspaces(what)


def _streaming_operands(seed=0, M=8, N=8192, K=4096):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(M, K, device="cuda", generator=g).bfloat16(), (torch.randn(N, K, device="cuda", generator=g) / 64).bfloat16()


def test_graphs_on_two_streams_share_nothing():
    """Two graphs (and a third with two branches) replayed side by side give the bits of one at a time; their workspaces come back when
    the graphs are gone."""
    import gc
    import time
    before = _used(1)
    ops = [_streaming_operands(i) for i in range(4)]
    want = [F.linear(x, w) for x, w in ops]
    graphs = []
    for i in range(2):
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            outs = [F.linear(*ops[i]) for _ in range(20)]
        graphs.append((graph, outs, want[i]))
    forked, side = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    with torch.cuda.graph(forked):
        side.wait_stream(torch.cuda.current_stream())
        a = [F.linear(*ops[2]) for _ in range(20)]
        with torch.cuda.stream(side):
            b = [F.linear(*ops[3]) for _ in range(20)]
        torch.cuda.current_stream().wait_stream(side)
    assert _used(1) == before + 4
    streams = [torch.cuda.Stream() for _ in range(3)]
    torch.cuda.synchronize()
    for _ in range(30):
        for s, g in zip(streams, [graphs[0][0], graphs[1][0], forked]):
            with torch.cuda.stream(s):
                g.replay()
    torch.cuda.synchronize()
    _lib.check_status()
    for _, outs, ref in graphs + [(forked, a, want[2]), (forked, b, want[3])]:
        assert all(torch.equal(o, ref) for o in outs)
    del graph, graphs, forked, outs, g, a, b, _
    gc.collect()
    torch.cuda.synchronize()
    for _ in range(50):                      # the driver lets go of a graph's objects on a thread of its own
        if _used(1) <= before:
            break
        time.sleep(0.1)
    assert _used(1) <= before


def test_every_stream_streams():
    """More streams than a process usually has: each takes the streaming form in a workspace of its own, and they may run side by side."""
    x, w = _streaming_operands(7)
    want = F.linear(x, w)
    held = _used(2)
    streams = [torch.cuda.Stream() for _ in range(12)]
    outs = []
    torch.cuda.synchronize()
    for _ in range(4):
        for s in streams:
            with torch.cuda.stream(s):
                outs.append(F.linear(x, w))
    torch.cuda.synchronize()
    _lib.check_status()
    assert all(torch.equal(o, want) for o in outs)
    assert held + 10 <= _used(2) <= held + 12 and _used(3) <= 512      # some of the pool's streams may have had one before


# 1408: skinny blocks of 8 + 8 columns, pairs of half tiles; 1000 and 8200: ragged tiles of 64 and 128 outputs, the up half right behind them;
# 24: less than a tile; 14336 x 4096: several blocks per tile, several tiles per block
@pytest.mark.parametrize("F_,K", [(1408, 512), (1000, 776), (8200, 264), (24, 64), (14336, 4096)])
@pytest.mark.parametrize("M", [1, 16, 40, 64, 65, 128, 131, 600])
def test_linear_glu(M, F_, K):
    x, w = torch.randn(M, K, device="cuda").bfloat16(), (torch.randn(2 * F_, K, device="cuda") * K ** -0.5).bfloat16()
    gu = x.double() @ w.double().t()
    for act, fn in (("swiglu", torch.nn.functional.silu), ("geglu", lambda v: torch.nn.functional.gelu(v, approximate="tanh"))):
        want = fn(gu[:, :F_]) * gu[:, F_:]
        y = F.linear_glu(x, w, act)
        torch.cuda.synchronize()
        _lib.check_status()
        e = _rel(y, want)
        # one rounding to bf16 (2^-9 at most, 2^-9 / sqrt(3) on average); through a rounded product three of them
        assert y.shape == (M, F_) and e < 4e-3
        assert e <= 1.05 * _rel(F.glu_fwd(F.gemm(x, w), act), want)
        assert torch.equal(y, F.linear_glu(x, w, act))


@pytest.mark.parametrize("B,S", [(1, 5), (2, 200)])
def test_scoring_without_gradients_matches_the_training_forward(B, S):
    """Without a gradient mode the blocks keep nothing and gate in the product; the logits are those of the pass that keeps everything."""
    from transformers_fusion_b200.models.config import TransformerConfig
    from transformers_fusion_b200.models.dense import DenseModel
    cfg = TransformerConfig(vocab_size=512, hidden_size=256, num_layers=2, num_heads=4, num_kv_heads=2, ffn_hidden_size=704, max_seq_len=256)
    m = DenseModel(cfg, device="cuda", dtype=torch.bfloat16, seed=0)
    ids = torch.randint(0, 512, (B, S), device="cuda")
    a = m(ids)
    with torch.no_grad():
        b = m(ids)
    assert a.requires_grad and not b.requires_grad and _rel(b, a.detach().double()) < 1e-2       # a few bf16 roundings per layer


def test_a_block_that_gives_up_leaves_the_counters_clear():
    """The bounds-check library lets one block's epilogue give up as if its wait had run out: the status word says so, and the products that
    follow (same and other shapes over the same counters) are right.  In a child process, because the library is chosen at load time."""
    import os
    import subprocess
    import sys
    code = r'''
import torch
from transformers_fusion_b200.ops import _lib, functional as F
_lib.register("tfb_test_rows_give_up", [_lib.c_i])
shapes = [(8, 4096, 4096), (3, 6144, 4096), (16, 28672, 512), (40, 8192, 2048)]
ops = [(torch.randn(M, K, device="cuda").bfloat16(), (torch.randn(N, K, device="cuda") * K ** -0.5).bfloat16()) for M, N, K in shapes]
def product(x, w):
    out = torch.full((x.shape[0], w.shape[0]), float("nan"), device="cuda")
    _lib.check(_lib.lib().tfb_gemm_rows(x.data_ptr(), x.stride(0), w.data_ptr(), w.stride(0), out.data_ptr(), out.stride(0), x.shape[0], w.shape[0],
                                        x.shape[1], None, None, 0, 1.0, 0, 1, 0, _lib.status_word().data_ptr(), _lib.stream()), "gemm_rows")
    return out
good = [product(x, w) for x, w in ops]
_lib.check_status()
for cta in (0, 3, 147):
    for x, w in ops:
        _lib.lib().tfb_test_rows_give_up(cta)
        product(x, w)
        _lib.lib().tfb_test_rows_give_up(-1)
        try:
            _lib.check_status()
            raise SystemExit("no status")
        except _lib.KernelError:
            pass
        for (a, b), want in zip(ops, good):
            assert torch.equal(product(a, b), want)
        _lib.check_status()
print("ok")
'''
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300, cwd=root, env=dict(os.environ, TFB_BOUNDS_CHECK="1"))
    assert r.returncode == 0 and "ok" in r.stdout, r.stdout[-1500:] + r.stderr[-1500:]
