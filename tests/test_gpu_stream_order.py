"""GPU tests of calls in a row on a context's stream: a call starts under the one before it, so that nothing may be read (weights,
keys, activations) or written before that one has completed. Expected bits are those of the same call on an idle stream."""
import ctypes as C
import math

import pytest

from fast_llm_b200 import capi
from fast_llm_b200.moe import MoeBlock

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def inputs(fmt, rows, cols, nx, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    blocks = rows * cols // capi.BLK_ELEMS[fmt]
    w = torch.randint(0, 256, (blocks, capi.BLK_BYTES[fmt]), dtype=torch.uint8, device="cuda", generator=g)
    d = (torch.rand(blocks, device="cuda", generator=g) * 0.01 + 0.001).half().view(torch.uint8).reshape(-1, 2)
    at = {capi.Q4_K: (0, 2), capi.Q6_K: (208,), capi.Q8_0: (0,)}[fmt]
    for o in at:
        w[:, o:o + 2] = d
    return w.reshape(rows, -1), torch.randn((nx, cols), device="cuda", generator=g)


class Writers:
    """What comes in front of a call here are kernels of the library's own that let the next launch start at their entry, behind a matvec
    whose last unit runs on one SM: the call's CTAs are on the other SMs before its inputs are written (an attention 8 us before the last
    of them, a matvec, which finds room only where the writers have left, 1.5 us)."""

    def __init__(self, ctx):
        self.ctx = ctx
        units = 2 * ctx.sm_count() + 1
        self.w, self.x = inputs(capi.Q4_K, 16 * units, 14336, 1, 77)
        self.y = torch.zeros(16 * units, device="cuda")

    def block(self):   # 14 us each where the call takes 5: the launches behind are all in the stream before these have run
        for _ in range(16):
            self.ctx.matvec_assign(capi.Q4_K, self.w, self.y.numel(), 14336, self.x, self.y)

    def fill(self, t, value):
        capi._ck(self.ctx.lib.fl_b200_memset(self.ctx._h, C.c_void_p(t.data_ptr()), value, C.c_size_t(t.numel() * t.element_size())))

    def floats(self, source, out):
        """out = source's weights times its column: random numbers that a matvec of the library writes."""
        w, x = source
        self.ctx.matvec_assign(capi.Q4_K, w, out.numel(), 2048, x, out)

    def source(self, n, seed, scale):
        w, x = inputs(capi.Q4_K, n, 2048, 1, seed)
        return w, x * scale

    def check(self, write, call, out):
        """call() after write(0), write(1), write(0), ... without a pause against the same one by one."""
        want = []
        for i in range(2):
            write(i, self.ctx.sync)
            call()
            self.ctx.sync()
            want.append([o.clone() for o in out])
        torch.cuda.synchronize()
        assert all(bool(torch.isfinite(o).all()) for w in want for o in w)
        assert not any(torch.equal(a, b) for a, b in zip(*want))
        got = []
        with torch.cuda.stream(torch.cuda.ExternalStream(self.ctx.stream())):
            for i in range(12):
                self.block()
                write(i % 2, lambda: None)
                call()
                call()
                got.append([o.clone() for o in out])
        torch.cuda.synchronize()
        for i, g in enumerate(got):
            assert all(torch.equal(a, b) for a, b in zip(g, want[i % 2])), i
        assert self.ctx.status() == 0


@pytest.mark.parametrize("n_tok,n_expert,top_k,n_ff", [(1, 4, 2, 2048), (4, 4, 2, 2048), (16, 8, 3, 4096), (19, 4, 1, 2048)])   # the last: two passes
def test_block_written_by_the_kernels_before(ctx, n_tok, n_expert, top_k, n_ff):
    E, wr = 2048, Writers(ctx)
    blk = MoeBlock(ctx, E, n_ff, n_expert, top_k, max_tokens=32)
    gate, up = (torch.zeros((n_expert * n_ff, capi.row_bytes(capi.Q4_K, E)), dtype=torch.uint8, device="cuda") for _ in range(2))
    down = torch.zeros((n_expert, E, capi.row_bytes(capi.Q4_K, n_ff)), dtype=torch.uint8, device="cuda")
    router, x = torch.zeros((n_expert, E), device="cuda"), torch.zeros((n_tok, E), device="cuda")
    y = [torch.zeros_like(x) for _ in range(2)]
    blk.set_weights(router, gate, up, down)
    xs, rs = ([wr.source(n, 10 * n + i, 0.01) for i in range(2)] for n in (n_tok * E, n_expert * E))
    torch.cuda.synchronize()

    def write(i, pause):   # every tensor of the block, the router last
        steps = [lambda: wr.fill(gate, 0x21 + i), lambda: wr.fill(up, 0x24 - i)]
        steps += [lambda e=e: wr.fill(down[e], 0x18 + e + 5 * i) for e in range(n_expert)]
        for s in steps + [lambda: wr.floats(xs[i], x), lambda: wr.floats(rs[i], router)]:
            s()
            pause()

    def call():   # another output each time: a call that repeats the one before it would be a replayed graph
        for o in y:
            blk.forward(x, n_tok, o)

    wr.check(write, call, y)
    blk.close()


# one position and several, with and without the records' sum; CTAs: one, one wave of one tile, of several, more than one wave; several positions on less
# than half the SMs, on more than half of them (one tile a CTA, several), on all
@pytest.mark.parametrize("kind,kv,batch,kv_len", [
    ("decode", 1, 1, 2), ("decode", 2, 1, 1024), ("lse", 1, 3, 20001), ("decode", 8, 16, 1100), ("lse", 8, 40, 64), ("verify", 1, 2, 100),
    ("verify", 1, 8, 30000), ("verify", 2, 8, 4000), ("verify", 2, 8, 16000), ("verify", 1, 16, 16000), ("verify", 8, 5, 9001)])
def test_attention_written_by_the_kernels_before(ctx, kind, kv, batch, kv_len):
    wr, shared = Writers(ctx), kind == "verify"
    seqs = 1 if shared else batch
    k, v = (torch.zeros((seqs * kv, kv_len, 128), dtype=torch.float16, device="cuda") for _ in range(2))
    q, out, lse = (torch.zeros((batch, 4 * kv, n), device="cuda") for n in (128, 128, 2))
    qs = [wr.source(q.numel(), 5 + i, 0.01) for i in range(2)]
    half, scale = kv_len // 2, 1.0 / math.sqrt(128)
    torch.cuda.synchronize()

    def write(i, pause):   # keys and values of the first half of the positions unlike those of the second, per head while there are few
        steps = [lambda: wr.floats(qs[i], q)]
        for t, first, rest in ((k, 0x2c + i, 0x30 - i), (v, 0x38 + i, 0x3c - 3 * i)):
            steps.append(lambda t=t, rest=rest: wr.fill(t, rest))
            steps += [lambda t=t, h=h, first=first: wr.fill(t[h, :half], first) for h in range(min(seqs * kv, 8))]
        for s in steps:
            s()
            pause()

    def call():
        if shared:
            ctx.attn_verify(q, k, v, 4 * kv, kv, 128, kv_len - batch + 1, kv_len, batch, scale, out)
        elif kind == "lse":
            ctx.attn_decode_lse(q, k, v, 4 * kv, kv, 128, kv_len, kv_len, batch, scale, out, lse)
        else:
            ctx.attn_decode(q, k, v, 4 * kv, kv, 128, kv_len, kv_len, batch, scale, out)

    wr.check(write, call, [out, lse] if kind == "lse" else [out])


# bytes that make numbers of a sane size in every format: scales of 0.01 to 0.07, quants and activations alike. A stage and a unit, several
# units a CTA, more columns than a thread converts at once; planes, slices of columns, two passes over the weights
@pytest.mark.parametrize("fmt", [capi.Q4_K, capi.Q6_K, capi.Q8_0])
@pytest.mark.parametrize("rows,cols,nx", [(16, 2048, 1), (4096, 4096, 1), (2049, 14336, 1), (4096, 4096, 3), (300, 2048, 16), (1000, 4096, 19)])
def test_matvec_written_by_the_kernels_before(ctx, fmt, rows, cols, nx):
    wr = Writers(ctx)
    w = torch.zeros((rows, capi.row_bytes(fmt, cols)), dtype=torch.uint8, device="cuda")
    x, y = torch.zeros((nx, cols), device="cuda"), torch.zeros((nx, rows), device="cuda")
    xs = [wr.source(nx * cols, 3 + i, 0.01) for i in range(2)]
    torch.cuda.synchronize()

    few = min(rows // 2, (1 << 20) // w.shape[1])   # a launch small enough to lie on the SMs beside the matvec in front

    def write(i, pause):   # the weights last, the rows of the first units last of all
        for s in (lambda: wr.floats(xs[i], x), lambda: wr.fill(w, 0x21 + i), lambda: wr.fill(w[:few], 0x2a - i)):
            s()
            pause()

    def call():
        if nx == 1:
            ctx.matvec_assign(fmt, w, rows, cols, x, y)
        else:
            wr.fill(y, 0)
            ctx.matvec(fmt, w, rows, cols, x, y, nx=nx, xstride=cols, ystride=rows)

    wr.check(write, call, [y])


@pytest.mark.parametrize("fmt", [capi.Q4_K, capi.Q6_K, capi.Q8_0])
def test_pitched_rows_written_by_the_kernels_before(ctx, fmt):
    rows, cols, wr = 1500, 2304, Writers(ctx)
    pitch = (capi.row_bytes(fmt, cols) + 15) // 16 * 16 + 16
    w, x, y = torch.zeros((rows, pitch), dtype=torch.uint8, device="cuda"), torch.zeros(cols, device="cuda"), torch.zeros(rows, device="cuda")
    xs = [wr.source(cols, 8 + i, 0.01) for i in range(2)]
    torch.cuda.synchronize()

    def write(i, pause):
        for s in (lambda: wr.floats(xs[i], x), lambda: wr.fill(w, 0x21 + i), lambda: wr.fill(w[:rows // 3], 0x2a - i)):
            s()
            pause()

    wr.check(write, lambda: ctx.matvec_pitched(fmt, w, rows, cols, pitch, x, y), [y])


def test_operands_written_on_the_legacy_default_stream(ctx):
    """The context's stream is a blocking one: a kernel on the legacy default stream lies between the calls in front of it and behind it."""
    rows = cols = 4096
    pair = [inputs(capi.Q4_K, rows, cols, 1, s) for s in (1, 2)]
    g = torch.Generator(device="cuda").manual_seed(5)
    kv = [tuple(torch.randn(4096 * 128, device="cuda", generator=g).half() for _ in range(2)) for _ in range(2)]
    w, x, y = torch.empty_like(pair[0][0]), torch.empty_like(pair[0][1]), torch.zeros(rows, device="cuda")
    k, v = torch.empty_like(kv[0][0]), torch.empty_like(kv[0][1])
    q, out = torch.randn((1, 4, 128), device="cuda", generator=g), torch.zeros((1, 4, 128), device="cuda")

    def call():
        ctx.matvec_assign(capi.Q4_K, w, rows, cols, x, y)
        ctx.attn_decode(q, k, v, 4, 1, 128, 4096, 4096, 1, 0.1, out)

    def write(i):
        for dst, src in zip((w, x, k, v), pair[i] + kv[i]):
            dst.copy_(src)

    want = []
    for i in range(2):
        write(i)
        torch.cuda.synchronize()
        call()
        ctx.sync()
        want.append((y.clone(), out.clone()))
    torch.cuda.synchronize()
    got = []
    for i in range(30):   # everything but the calls on the default stream, nothing waited for
        write(i % 2)
        call()
        got.append((y.clone(), out.clone()))
    torch.cuda.synchronize()
    assert not torch.equal(want[0][0], want[1][0]) and not torch.equal(want[0][1], want[1][1])
    assert all(torch.equal(a, b) for i, pair in enumerate(got) for a, b in zip(pair, want[i % 2]))


@pytest.mark.parametrize("fmt", [capi.Q4_K, capi.Q6_K, capi.Q8_0])
@pytest.mark.parametrize("rows,cols,nx", [(16, 2048, 1), (4096, 4096, 1), (2049, 14336, 1), (4096, 4096, 3), (300, 2048, 16)])
def test_weights_written_by_the_kernel_before(ctx, fmt, rows, cols, nx):
    pair = [inputs(fmt, rows, cols, nx, s) for s in (1, 2)]
    w, x = torch.empty_like(pair[0][0]), torch.empty_like(pair[0][1])
    y = torch.zeros((nx, rows), device="cuda")

    def call():
        if nx == 1:
            ctx.matvec_assign(fmt, w, rows, cols, x, y)
        else:
            capi._ck(ctx.lib.fl_b200_memset(ctx._h, C.c_void_p(y.data_ptr()), 0, C.c_size_t(4 * nx * rows)))
            ctx.matvec(fmt, w, rows, cols, x, y, nx=nx, xstride=cols, ystride=rows)

    want = []
    for a, b in pair:
        w.copy_(a)
        x.copy_(b)
        torch.cuda.synchronize()
        call()
        ctx.sync()
        want.append(y.clone())
    assert not torch.equal(*want)
    torch.cuda.synchronize()
    got = []
    with torch.cuda.stream(torch.cuda.ExternalStream(ctx.stream())):
        zero = torch.zeros_like(w[:1])
        for i in range(40):   # kernels that write weights and activation, the call, a kernel that reads its result
            a, b = pair[i % 2]
            torch.bitwise_or(a, zero, out=w)
            torch.mul(b, 1.0, out=x)
            call()
            call()
            got.append(y.clone())
    torch.cuda.synchronize()
    assert all(torch.equal(g, want[i % 2]) for i, g in enumerate(got))
    assert ctx.status() == 0


@pytest.mark.parametrize("kv_len,batch", [(1, 1), (1024, 1), (4097, 3)])
def test_cache_written_by_the_kernel_before(ctx, kv_len, batch):
    g = torch.Generator(device="cuda").manual_seed(kv_len)
    pair = [tuple(torch.randn(s, device="cuda", generator=g).to(t) for s, t in (((batch, 8, 128), torch.float32), ((batch, 2, kv_len, 128), torch.float16),
                                                                              ((batch, 2, kv_len, 128), torch.float16))) for _ in range(2)]
    q, k, v = (torch.empty_like(t) for t in pair[0])
    out = torch.zeros_like(q)

    def call():
        ctx.attn_decode(q, k, v, 8, 2, 128, kv_len, kv_len, batch, 1.0 / math.sqrt(128), out)

    want = []
    for p in pair:
        for dst, src in zip((q, k, v), p):
            dst.copy_(src)
        torch.cuda.synchronize()
        call()
        ctx.sync()
        want.append(out.clone())
    torch.cuda.synchronize()
    got = []
    with torch.cuda.stream(torch.cuda.ExternalStream(ctx.stream())):
        for i in range(40):
            for dst, src in zip((q, k, v), pair[i % 2]):
                torch.mul(src, 1.0, out=dst)
            call()
            call()
            got.append(out.clone())
    torch.cuda.synchronize()
    assert all(torch.equal(o, want[i % 2]) for i, o in enumerate(got))


@pytest.mark.parametrize("offset,size", [(0, 1), (0, 16), (1, 15), (3, 14), (15, 1), (7, 4096), (16, 4099), (5, 3_000_001), (0, 64 << 20),
                                         (1, 128 << 20), (1, (128 << 20) + 1)])   # the largest of the library's own kernel, the driver's
def test_memset_any_range(ctx, offset, size):
    buf = torch.randint(0, 200, (offset + size + 40,), dtype=torch.uint8, device="cuda")
    want = buf.clone()
    want[offset:offset + size] = 0xAB
    torch.cuda.synchronize()
    capi._ck(ctx.lib.fl_b200_memset(ctx._h, C.c_void_p(buf.data_ptr() + offset), 0x1AB, C.c_size_t(size)))   # the low byte, as memset
    ctx.sync()
    assert torch.equal(buf, want)


def test_memset_what_the_driver_takes_or_refuses(ctx):
    host = torch.full((100,), 7, dtype=torch.uint8).pin_memory()
    capi._ck(ctx.lib.fl_b200_memset(ctx._h, C.c_void_p(host.data_ptr()), 1, C.c_size_t(100)))
    capi._ck(ctx.lib.fl_b200_memset(ctx._h, C.c_void_p(0), 0, C.c_size_t(0)))
    ctx.sync()
    assert bool((host == 1).all())
    assert ctx.lib.fl_b200_memset(ctx._h, C.c_void_p(0), 0, C.c_size_t(16)) != 0   # no memory there: refused, nothing is launched
    ctx.sync()
