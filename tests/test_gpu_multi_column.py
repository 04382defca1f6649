"""GPU tests of the multi-column matmul (csrc/matvec_tc_nx.cu), of its grouped form and of the attention of several positions
over one cache (csrc/attn.cu: attn_shared_kernel) at the edges of their dispatch, against f64 arithmetic on the same
quantised weights (dequantisation itself is tested bit for bit elsewhere).

Tolerance of a matmul: a result is a sum of n = columns / 256 super-blocks, each a chain of f32 additions (at most 16
tensor-core steps, which truncate, and about ten rounded ones), with operands exact to 2^-22. The error of a sum is that
of its terms' size, not of the result's: 16 * 2^-23 + 2^-22 per super-block, the super-blocks' errors independent, hence
about 2.2e-6 * sum |w x| / sqrt(n) at worst; measured 1e-7 .. 6e-7 of the result's root mean square. The bound used is
1e-5 of the root mean square of the exact result, below what a single wrong weight of a row changes."""
import math

import numpy as np
import pytest

from fast_llm_b200 import capi, synth
from fast_llm_b200.moe import MoeBlock

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def weights(ctx, fmt, rows, cols, seed):
    w = torch.from_numpy(synth.quant_tensor(fmt, np.random.default_rng(seed), rows, cols)).cuda()
    f = torch.empty((rows, cols), device="cuda")
    torch.cuda.synchronize()
    ctx.dequant(fmt, w, rows, cols, f)
    ctx.sync()
    return w, f.double()


def close(got, want, tol=1e-5):
    want = want.double()
    return float((got.double() - want).abs().max() / (want.pow(2).mean().sqrt() + 1e-300)) <= tol


CASES = [(fmt, 100, 4096, nx) for fmt in (capi.Q4_K, capi.Q6_K, capi.Q8_0) for nx in (2, 4, 5, 8, 9, 12, 13, 16, 17, 33)]
CASES += [
    (capi.Q4_K, 1, 256, 2), (capi.Q6_K, 15, 2048, 3), (capi.Q8_0, 17, 256, 16),      # fewer rows than a unit, one block
    (capi.Q4_K, 33, 768, 7), (capi.Q8_0, 33, 768, 7), (capi.Q4_K, 50, 2304, 16),     # rows that are no whole swizzle lines
    (capi.Q8_0, 40, 3072, 11), (capi.Q8_0, 40, 1280, 6),                             # second half of a Q8_0 segment empty
    (capi.Q4_K, 64, 18432, 16), (capi.Q6_K, 64, 18432, 16), (capi.Q8_0, 64, 18432, 16),   # the most parts
    (capi.Q4_K, 64, 8192, 4), (capi.Q6_K, 48, 14336, 8), (capi.Q8_0, 48, 14336, 3),
    (capi.Q4_K, 131072, 4352, 16),   # more rows than the planes of partial results hold: slices
]


@pytest.mark.parametrize("fmt,rows,cols,nx", CASES)
def test_multi_column_edges(ctx, fmt, rows, cols, nx):
    w, f = weights(ctx, fmt, rows, cols, rows + cols + nx)
    gen = torch.Generator(device="cuda").manual_seed(nx)
    x = torch.full((nx, cols + 8), float("nan"), device="cuda")   # the gap between columns is never read
    x[:, :cols] = torch.randn((nx, cols), device="cuda", generator=gen) * torch.logspace(-3, 3, nx, device="cuda")[:, None]
    y = torch.randn((nx, rows + 3), device="cuda", generator=gen)   # rows of no multiple of 16 bytes
    want = y.double()
    want[:, :rows] += x[:, :cols].double() @ f.T
    torch.cuda.synchronize()
    ctx.matvec(fmt, w, rows, cols, x, y, nx=nx, xstride=cols + 8, ystride=rows + 3)
    ctx.sync()
    assert ctx.status() == 0
    for p in range(nx):
        assert close(y[p, :rows], want[p, :rows]), "column %d" % p
        assert torch.equal(y[p, rows:].double(), want[p, rows:]), "written past the rows of column %d" % p


@pytest.mark.parametrize("fmt", [capi.Q4_K, capi.Q6_K, capi.Q8_0])
def test_multi_column_special_values(ctx, fmt):
    """Zero columns, the smallest and largest magnitudes, one outlier per column; a column that holds an infinity or a NaN
    spoils its own results only."""
    rows, cols, nx = 64, 2048, 8
    w, f = weights(ctx, fmt, rows, cols, 3)
    x = torch.randn((nx, cols), device="cuda", generator=torch.Generator(device="cuda").manual_seed(1))
    x[1] = 0
    x[2] *= 1e-30
    x[3] *= 1e25
    x[4, 700] = 1e6
    x[5, 9] = float("inf")
    x[6, 2047] = float("nan")
    y = torch.zeros((nx, rows), device="cuda")
    torch.cuda.synchronize()
    ctx.matvec(fmt, w, rows, cols, x, y, nx=nx, xstride=cols, ystride=rows)
    ctx.sync()
    assert torch.equal(y[1], torch.zeros_like(y[1]))
    for p in (0, 2, 3, 4, 7):
        assert close(y[p], f @ x[p].double()), "column %d" % p
    assert not torch.isfinite(y[5]).any() and torch.isnan(y[6]).all()


def centred_q4k(rows, cols, seed):
    """Q4_K as trained tensors have it: zero mean, every min 7.5 steps of its scale."""
    gen, nb = torch.Generator(device="cuda").manual_seed(seed), rows * cols // 256
    w = torch.randint(0, 256, (nb, 144), dtype=torch.uint8, device="cuda", generator=gen)
    d = (torch.rand((nb, 1), device="cuda", generator=gen) * 0.4 + 0.8) / (220.0 * math.sqrt(cols))
    w[:, 0:2], w[:, 2:4] = ((d * s).half().view(torch.uint8).reshape(nb, 2) for s in (1.0, 7.5))
    sc = torch.randint(32, 64, (nb, 8), dtype=torch.uint8, device="cuda", generator=gen)
    w[:, 4:8] = w[:, 8:12] = sc[:, :4] | ((sc[:, 4:] >> 4) << 6)
    w[:, 12:16] = (sc[:, 4:] & 15) * 17
    return w.reshape(rows, -1)


@pytest.mark.parametrize("nx", [4, 8, 16])
def test_q4_k_sums_are_not_truncated(ctx, nx):
    """mma.sync truncates its running sum towards zero: half a unit, 2^-25 to 2^-24 of it, per instruction on average and
    always towards zero. Chains of 4 from zero, whose sum reaches its size on the way only, lose some 6e-8 of every result
    (measured 5.5e-8; chains of 8: 1.0e-7), beside errors of random sign that leave 1.2e-7 in all (chains of 8: 1.7e-7)."""
    rows = cols = 4096
    w = centred_q4k(rows, cols, nx)
    f = torch.empty((rows, cols), device="cuda")
    x = torch.randn((nx, cols), device="cuda", generator=torch.Generator(device="cuda").manual_seed(nx))
    y = torch.zeros((nx, rows), device="cuda")
    torch.cuda.synchronize()
    ctx.dequant(capi.Q4_K, w, rows, cols, f)
    ctx.matvec(capi.Q4_K, w, rows, cols, x, y, nx=nx, xstride=cols, ystride=rows)
    ctx.sync()
    want = x.double() @ f.double().T
    assert abs(float((y.double() * want).sum() / want.pow(2).sum()) - 1) <= 8e-8
    assert float((y.double() - want).norm() / want.norm()) <= 1.5e-7


@pytest.mark.parametrize("fmt_gu,fmt_d,n_expert,top_k,n_tok,max_tokens", [
    (capi.Q4_K, capi.Q4_K, 8, 2, 16, 16), (capi.Q4_K, capi.Q6_K, 16, 1, 3, 16), (capi.Q6_K, capi.Q4_K, 4, 4, 16, 16),
    (capi.Q4_K, capi.Q4_K, 4, 3, 45, 64),    # more tokens per expert than a pass takes
    (capi.Q4_K, capi.Q4_K, 64, 1, 2, 16),    # most experts idle
    (capi.Q4_K, capi.Q4_K, 48, 6, 16, 16),   # more than 32 at work: the conversion's lookup takes a second round
])
def test_grouped_experts(ctx, fmt_gu, fmt_d, n_expert, top_k, n_tok, max_tokens):
    E, F = 2048, 4096
    blk = MoeBlock(ctx, E, F, n_expert, top_k, norm=1, scale=1.0, fmt_gate_up=fmt_gu, fmt_down=fmt_d, max_tokens=max_tokens)
    (wg, fg), (wu, fu), (wd, fd) = (weights(ctx, fmt, n_expert * r, c, s)
                                    for fmt, r, c, s in ((fmt_gu, F, E, 1), (fmt_gu, F, E, 2), (fmt_d, E, F, 3)))
    gen = torch.Generator(device="cuda").manual_seed(n_tok)
    router = torch.randn((n_expert, E), device="cuda", generator=gen)
    x = torch.randn((n_tok, E), device="cuda", generator=gen)
    y = torch.zeros_like(x)
    blk.set_weights(router, wg, wu, wd)
    torch.cuda.synchronize()
    for _ in range(3):   # direct, recorded, replayed
        y.zero_()
        torch.cuda.synchronize()
        blk.forward(x, n_tok, y)
        ctx.sync()
        assert ctx.status() == 0
    p = torch.softmax(x.double() @ router.double().T, dim=-1)
    top, ids = torch.topk(p, top_k, dim=-1)
    top = top / top.sum(-1, keepdim=True)
    want = torch.zeros((n_tok, E), dtype=torch.float64, device="cuda")
    for t in range(n_tok):
        for g, e in zip(top[t], ids[t].tolist()):
            h = torch.nn.functional.silu(fg[e * F:(e + 1) * F] @ x[t].double()) * (fu[e * F:(e + 1) * F] @ x[t].double())
            want[t] += g * (fd[e * E:(e + 1) * E] @ h)
    # silu and the products multiply the relative errors of three matmuls and of the gate
    assert close(y, want, 1e-4)


@pytest.mark.parametrize("n_tok", [1, 2, 16])
@pytest.mark.parametrize("fmt", [capi.Q4_K, capi.Q6_K])
def test_block_of_experts_precision(ctx, fmt, n_tok):
    """A block called by itself, one token like several: activations of 22 bits, f32 sums. Gate, up and down of weights of zero
    mean are each some 1.2e-7 off (2-norm), a share of it the truncation that all three have with the same sign; the product
    of gate and up has both errors; together 2.1e-7 to 3.7e-7. (Activations of 21 bits per 256 columns: 2.3e-6.)"""
    E, F, n, k = 2048, 2048, 4, 1
    blk = MoeBlock(ctx, E, F, n, k, norm=1, scale=1.0, fmt_gate_up=fmt, fmt_down=fmt, max_tokens=16)
    ws, fs = [], []
    for i, (r, c) in enumerate(((n * F, E), (n * F, E), (n * E, F))):
        if fmt == capi.Q4_K:
            ws.append(centred_q4k(r, c, i))
            fs.append(torch.empty((r, c), device="cuda"))
            torch.cuda.synchronize()
            ctx.dequant(fmt, ws[-1], r, c, fs[-1])
            ctx.sync()
            fs[-1] = fs[-1].double()
        else:
            w, f = weights(ctx, fmt, r, c, i)
            ws.append(w)
            fs.append(f)
    gen = torch.Generator(device="cuda").manual_seed(n_tok)
    router, x = torch.randn((n, E), device="cuda", generator=gen), torch.randn((n_tok, E), device="cuda", generator=gen)
    y = torch.zeros_like(x)
    blk.set_weights(router, *ws)
    torch.cuda.synchronize()
    blk.forward(x, n_tok, y)
    ctx.sync()
    assert ctx.status() == 0
    want, xd = torch.zeros((n_tok, E), dtype=torch.float64, device="cuda"), x.double()
    for t, e in enumerate((xd @ router.double().T).argmax(-1).tolist()):
        g, u = (f[e * F:(e + 1) * F] @ xd[t] for f in fs[:2])
        want[t] = fs[2][e * E:(e + 1) * E] @ (torch.nn.functional.silu(g) * u)
    assert float((y.double() - want).norm() / want.norm()) <= 4.3e-7


def test_block_of_experts_memory(ctx):
    """What a block holds besides a row of results per (token, slot) pair does not grow with max_tokens and is shared by the
    blocks of a context: creating one for many tokens takes less than two rows of n_ff and one of n_embd floats per pair, and
    the sixteenth block of 16 tokens next to nothing."""
    E, F, k = 4096, 14336, 2

    def free():
        ctx.sync()
        return torch.cuda.mem_get_info()[0]
    before = free()
    big = MoeBlock(ctx, E, F, 8, k, max_tokens=2048)
    assert before - free() <= 2048 * k * 4 * (2 * F + E)
    big.close()
    assert before - free() <= 1 << 21   # given back
    blocks = [MoeBlock(ctx, E, F, 8, k, max_tokens=16) for _ in range(16)]
    assert before - free() <= 16 * 16 * k * 4 * (2 * F + E)
    for b in blocks:
        b.close()
    assert before - free() <= 1 << 21


def test_blocks_of_experts_share_scratch(ctx):
    """Blocks of different sizes and formats called in turn, directly and as recorded launches, and after the largest has gone:
    every result is what the block gives alone."""
    shapes = [(2048, 2048, 4, 2, capi.Q4_K, 16, 5), (2048, 4096, 8, 2, capi.Q6_K, 64, 40), (4096, 2048, 4, 1, capi.Q4_K, 16, 16)]
    blocks, args, alone = [], [], []
    for i, (E, F, n, k, fmt, max_tokens, n_tok) in enumerate(shapes):
        ws = [weights(ctx, fmt, r, c, 10 * i + j)[0] for j, (r, c) in enumerate(((n * F, E), (n * F, E), (n * E, F)))]
        gen = torch.Generator(device="cuda").manual_seed(i)
        router, x = torch.randn((n, E), device="cuda", generator=gen), torch.randn((n_tok, E), device="cuda", generator=gen)
        first = MoeBlock(ctx, E, F, n, k, fmt_gate_up=fmt, fmt_down=fmt, max_tokens=max_tokens)
        y = torch.zeros_like(x)
        first.set_weights(router, *ws)
        torch.cuda.synchronize()
        first.forward(x, n_tok, y)
        ctx.sync()
        first.close()
        alone.append(y)
        args.append((router, ws, x, n_tok))
    for (E, F, n, k, fmt, max_tokens, n_tok), (router, ws, x, _) in zip(shapes, args):
        blocks.append(MoeBlock(ctx, E, F, n, k, fmt_gate_up=fmt, fmt_down=fmt, max_tokens=max_tokens))
        blocks[-1].set_weights(router, *ws)
    outs = [torch.zeros_like(y) for y in alone]
    for turn in range(4):
        if turn == 3:
            blocks.pop(1).close()
            del outs[1], args[1], alone[1]
        for y in outs:
            y.zero_()
        torch.cuda.synchronize()
        for b, (_, _, x, n_tok), y in zip(blocks, args, outs):
            b.forward(x, n_tok, y)
        ctx.sync()
        assert ctx.status() == 0
        for y, want in zip(outs, alone):
            assert torch.equal(y, want)


@pytest.mark.parametrize("n_draft", [2, 3, 7, 8, 9, 16])
@pytest.mark.parametrize("base", [1, 40, 63, 64, 65, 500, 4100])
def test_shared_cache_positions(ctx, base, n_draft):
    """Position b attends base + b keys; the cache rows behind the last one hold NaN."""
    H, stride = 3, base + n_draft + 70
    gen = torch.Generator(device="cuda").manual_seed(base * 31 + n_draft)
    k, v = (torch.full((H, stride, 128), float("nan"), dtype=torch.float16, device="cuda") for _ in "kv")
    n = base + n_draft - 1
    for c in (k, v):
        c[:, :n] = torch.randn((H, n, 128), device="cuda", generator=gen).half()
    q = torch.randn((n_draft, 4 * H, 128), device="cuda", generator=gen) * 2
    out = torch.zeros_like(q)
    torch.cuda.synchronize()
    ctx.attn_verify(q, k, v, 4 * H, H, 128, base, stride, n_draft, 1 / math.sqrt(128), out)
    ctx.sync()
    assert ctx.status() == 0
    for b in range(n_draft):
        kk, vv = (c[:, :base + b].double().repeat_interleave(4, dim=0) for c in (k, v))
        p = torch.softmax(torch.einsum("hd,hkd->hk", q[b].double(), kk) / math.sqrt(128), dim=-1)
        want = torch.einsum("hk,hkd->hd", p, vv)
        # probabilities and q are exact to 2^-22, sums f32; expf is within 2 ulp: a few 1e-6 of the context's size
        assert float((out[b].double() - want).abs().max()) <= 2e-5


@pytest.mark.parametrize("base,n_draft,bad", [(60, 4, 2), (1, 8, 3), (58, 8, 5), (500, 16, 9), (4090, 16, 7), (4090, 2, 1)])
def test_shared_cache_rows_of_later_positions(ctx, base, n_draft, bad):
    """The rows of positions `bad` and later hold infinities and NaN: the positions in front of them, which do not attend those
    rows, are what they are without."""
    H, n = 2, base + n_draft - 1
    gen = torch.Generator(device="cuda").manual_seed(base + n_draft)
    k, v = (torch.randn((H, n, 128), device="cuda", generator=gen).half() for _ in "kv")
    q = torch.randn((n_draft, 4 * H, 128), device="cuda", generator=gen) * 2
    want, out = torch.zeros_like(q), torch.zeros_like(q)
    torch.cuda.synchronize()
    ctx.attn_verify(q, k, v, 4 * H, H, 128, base, n, n_draft, 1 / math.sqrt(128), want)
    ctx.sync()
    row = base + bad - 1   # the first row that position `bad` attends and position bad - 1 does not
    v[:, row] = float("inf")
    v[:, row + 1:] = float("nan")
    k[:, row, ::2] = float("-inf")
    k[:, row + 1:] = float("nan")
    torch.cuda.synchronize()
    ctx.attn_verify(q, k, v, 4 * H, H, 128, base, n, n_draft, 1 / math.sqrt(128), out)
    ctx.sync()
    assert ctx.status() == 0
    assert torch.isfinite(want).all()
    assert torch.equal(out[:bad], want[:bad])   # the same sums in the same order, bit for bit


@pytest.mark.parametrize("n_draft", [2, 8])
def test_shared_cache_long_context_sums(ctx, n_draft):
    """The sums over many keys are rounded, not truncated. Scores and probabilities carry 2^-22 and expf 2 ulp, independent
    from key to key; measured 4.5e-7 (2-norm) at 4096 as at 65536 keys. A running sum truncated at every step: 1.5e-6."""
    H, n = 2, 65536
    gen = torch.Generator(device="cuda").manual_seed(n_draft)
    k, v = (torch.randn((H, n, 128), device="cuda", generator=gen).half() for _ in "kv")
    q = torch.randn((n_draft, 4 * H, 128), device="cuda", generator=gen)
    out = torch.zeros_like(q)
    torch.cuda.synchronize()
    ctx.attn_verify(q, k, v, 4 * H, H, 128, n - n_draft + 1, n, n_draft, 1 / math.sqrt(128), out)
    ctx.sync()
    for b in range(n_draft):
        kk, vv = (c[:, :n - n_draft + 1 + b].double().repeat_interleave(4, dim=0) for c in (k, v))
        want = torch.einsum("hk,hkd->hd", torch.softmax(torch.einsum("hd,hkd->hk", q[b].double(), kk) / math.sqrt(128), dim=-1), vv)
        assert float((out[b].double() - want).norm() / want.norm()) <= 8e-7, b


@pytest.mark.parametrize("rows,cols", [(16, 256), (512, 2304), (48, 14336)])
def test_expert_rows_one_column(ctx, rows, cols):
    """One column of a device-side expert: the last expert of the stack, and the mark that makes the launch leave its output
    alone."""
    n = 5
    w, f = weights(ctx, capi.Q4_K, n * rows, cols, rows + cols)
    x = torch.randn(cols, device="cuda", generator=torch.Generator(device="cuda").manual_seed(2))
    idx = torch.zeros(1, dtype=torch.int32, device="cuda")
    for e in (n - 1, 0, -1):
        y = torch.full((rows,), 3.0, device="cuda")
        idx.fill_(e)
        torch.cuda.synchronize()
        ctx.matvec_expert(capi.Q4_K, w, rows, cols, idx, rows * capi.row_bytes(capi.Q4_K, cols), x, y)
        ctx.sync()
        assert ctx.status() == 0
        if e < 0:
            assert torch.equal(y, torch.full_like(y, 3.0))
        else:
            assert close(y - 3.0, f[e * rows:(e + 1) * rows] @ x.double(), 2e-5)


@pytest.mark.parametrize("rows,cols", [(1, 256), (33, 1024), (100, 2304), (64, 3072), (40, 14336)])
def test_q8_0_one_column(ctx, rows, cols):
    """Q8_0 on the tensor-core kernel, with extreme quants and one outlier in the activation."""
    w, _ = weights(ctx, capi.Q8_0, rows, cols, rows + cols)
    blk = w.view(-1, 34)
    blk[0, 2:] = 0x80                        # -128
    blk[-1, 2:] = 0x7F
    f = torch.empty((rows, cols), device="cuda")
    torch.cuda.synchronize()
    ctx.dequant(capi.Q8_0, w, rows, cols, f)
    x = torch.randn(cols, device="cuda", generator=torch.Generator(device="cuda").manual_seed(4))
    x[cols // 2] = 1e4
    y = torch.zeros(rows, device="cuda")
    torch.cuda.synchronize()
    ctx.matvec_assign(capi.Q8_0, w, rows, cols, x, y)
    ctx.sync()
    assert close(y, f.double() @ x.double())
