"""The fused form (decomposition + forward column pass, row pass on the pair layout, inverse column
pass + CRT; the 16-row split) against the plain form of the same point, whose kernels share none of
its code, at the edges of its ranges.  Results are integers: every byte must be equal."""
import numpy as np
import pytest

from conftest import ensure_library, orc

pytestmark = pytest.mark.gpu


def _torch():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


def _q(N, W):
    """Largest number below 2^W that is 1 mod 2N (the library needs no primality)."""
    return (1 << W) - 2 * N + 1


def _operands(torch, N, W, count, seed, off):
    """[count, N, L] operands below q, `off` words past a 256-byte boundary; the largest value in
    a few coefficients."""
    L = (W + 31) // 32
    rng = np.random.default_rng(seed)
    x = rng.integers(0, 1 << 32, size=(count, N, L), dtype=np.uint64).astype(np.uint32)
    if W % 32:
        x[..., -1] &= np.uint32((1 << (W % 32)) - 1)
    x[..., -1] &= np.uint32(~(1 << ((W - 1) % 32)) & 0xFFFFFFFF)  # below 2^(W-1) < q
    x[:, [0, 1, N // 2, N - 1]] = orc.limbs_of(_q(N, W) - 1, L)
    buf = torch.zeros(x.size + 64, dtype=torch.int32, device="cuda")
    v = buf[off:off + x.size].view(count, N, L)
    v.copy_(torch.from_numpy(x.view(np.int32)))
    return x, v


# primes K around the lane groups (32 / 33, 64 / 65 and the largest), limb counts of every residue
# mod 4, the shortest and longest rows, tile counts that leave lane groups of a super-tile empty,
# and more tiles than one round of CTAs; (512, 1820) is the first point past the fused CRT's shared
# memory (more than 120 primes) and runs the separate passes
POINTS = [(512, 64, 1), (512, 470, 3), (512, 476, 5), (1024, 948, 2), (1024, 956, 1), (512, 1786, 3), (512, 1820, 3), (2048, 97, 40),
          (2048, 130, 7), (4096, 256, 33), (8192, 1001, 3), (16384, 300, 9), (32768, 868, 2), (65536, 64, 3),
          (65536, 1747, 2)]


@pytest.mark.parametrize("N,W,count", POINTS)
@pytest.mark.parametrize("off", [0, 1])
def test_fused_form_equals_plain_form(N, W, count, off):
    torch = _torch()
    import polymult
    ensure_library()
    L = (W + 31) // 32
    q = orc.limbs_of(_q(N, W), L)
    _, a = _operands(torch, N, W, count, N + W, off)
    _, b = _operands(torch, N, W, count, N + W + 1, 0)
    s = torch.cuda.current_stream().cuda_stream
    out = {}
    for gemm in ("tensor", "plain"):
        c = torch.full((count, N, L), -1, dtype=torch.int32, device="cuda")
        with polymult.Multiplier(N, W, q, gemm=gemm) as m:
            if gemm == "tensor":
                assert m.info()["launches_per_multiply"] == (3 if W < 1800 else 7)
            m.multiply_device(a.data_ptr(), b.data_ptr(), c.data_ptr(), count, s)
            m.sync()
        out[gemm] = c
    assert torch.equal(out["tensor"], out["plain"])


@pytest.mark.parametrize("body", [1, 4, 16])
@pytest.mark.parametrize("N,W", [(512, 200), (1024, 64), (4096, 300)])
def test_host_chunks_of_any_width(N, W, body):
    """Column chunks of whole 8-column tiles run the fused kernels, narrower ones the separate
    passes (N = 1024 in sixteenths: two columns from an odd one on); the products are the same."""
    torch = _torch()
    import polymult
    ensure_library()
    L = (W + 31) // 32
    xa, a = _operands(torch, N, W, 1, 5, 0)
    xb, b = _operands(torch, N, W, 1, 6, 0)
    c = torch.zeros((1, N, L), dtype=torch.int32, device="cuda")
    with polymult.Multiplier(N, W, orc.limbs_of(_q(N, W), L), gemm="tensor") as m:
        m.multiply_device(a.data_ptr(), b.data_ptr(), c.data_ptr(), 1, torch.cuda.current_stream().cuda_stream)
        m.sync()
        m.set_pipeline(body, body)
        got = m.multiply(xa[0], xb[0])
    assert np.array_equal(got, c.cpu().numpy().view(np.uint32)[0])


@pytest.mark.parametrize("N,W,gemm", [(512, 300, "tensor"), (512, 128, "tensor"), (256, 300, "tensor"), (512, 3000, "tensor"),
                                      (512, 300, "plain")])
def test_reduction_at_its_carries(N, W, gemm):
    """a = 1: the products are b's coefficients, chosen so that the reduction's sums carry out of the
    low limbs (runs of ones of every length, values next to q and to multiples of 2^32)."""
    torch = _torch()
    import polymult
    ensure_library()
    L = (W + 31) // 32
    q = _q(N, W)
    vals = [(1 << k) - 1 for k in range(1, W)] + [(1 << W) - 1 - (1 << k) for k in range(2 * N.bit_length(), W)]
    vals += [q - 1 - k for k in range(40)] + [1 << k for k in range(W - 1)]
    vals = [v for v in vals if v < q]
    a = np.zeros((N, L), dtype=np.uint32)
    a[0, 0] = 1
    s = torch.cuda.current_stream().cuda_stream
    da = torch.from_numpy(a.view(np.int32)).cuda()
    with polymult.Multiplier(N, W, orc.limbs_of(q, L), gemm=gemm) as m:
        for i in range(0, len(vals), N):
            part = vals[i:i + N]
            b = np.zeros((N, L), dtype=np.uint32)
            for k, v in enumerate(part):
                b[k] = orc.limbs_of(v, L)
            db = torch.from_numpy(b.view(np.int32)).cuda()
            c = torch.zeros_like(db)
            m.multiply_device(da.data_ptr(), db.data_ptr(), c.data_ptr(), 1, s)
            m.sync()
            assert torch.equal(c, db)


@pytest.mark.parametrize("N,W", [(512, 300), (512, 3000), (4096, 256)])
def test_call_between_other_kernels_of_its_stream(N, W):
    """The first launch of a call may start under the kernel before it: operands written by that
    kernel, and overwritten by the one after the call, give the products of calls run one by one."""
    torch = _torch()
    import polymult
    ensure_library()
    L = (W + 31) // 32
    _, xs = _operands(torch, N, W, 6, 8, 0)
    _, b = _operands(torch, N, W, 1, 9, 0)
    s = torch.cuda.current_stream().cuda_stream
    with polymult.Multiplier(N, W, orc.limbs_of(_q(N, W), L), gemm="tensor") as m:
        def run(a, c):
            m.multiply_device(a.data_ptr(), b.data_ptr(), c.data_ptr(), 1, s)
        want = []
        for i in range(6):
            c = torch.zeros((N, L), dtype=torch.int32, device="cuda")
            torch.cuda.synchronize()
            run(xs[i], c)
            m.sync()
            want.append(c)
        a, c = torch.zeros_like(xs[0]), torch.zeros_like(xs[0])
        got = [torch.zeros_like(a) for _ in range(6)]
        for i in range(6):
            torch.bitwise_or(xs[i], 0, out=a)
            run(a, c)
            torch.bitwise_or(c, 0, out=got[i])
            a.fill_(-1)
        m.sync()
    for g, w in zip(got, want):
        assert torch.equal(g, w)


@pytest.mark.parametrize("L0", [1, 9, 17, 25, 33, 41, 49])
def test_every_limb_count(L0):
    """The CRT's epilogue takes a coefficient's limbs in halves, pairs of four-limb steps, a step left
    over and up to three limbs behind it: every limb count of the fused form, so that each of these
    endings is met by both halves."""
    torch = _torch()
    import polymult
    ensure_library()
    N, s = 512, torch.cuda.current_stream().cuda_stream
    for L in range(L0, min(L0 + 8, 57)):
        W = 32 * L - 13
        _, a = _operands(torch, N, W, 2, 3 * L, 0)
        _, b = _operands(torch, N, W, 2, 3 * L + 1, 0)
        out = []
        for gemm in ("tensor", "plain"):
            c = torch.full((2, N, L), -1, dtype=torch.int32, device="cuda")
            with polymult.Multiplier(N, W, orc.limbs_of(_q(N, W), L), gemm=gemm) as m:
                if gemm == "tensor":
                    assert m.info()["launches_per_multiply"] == 3
                m.multiply_device(a.data_ptr(), b.data_ptr(), c.data_ptr(), 2, s)
                m.sync()
            out.append(c)
        assert torch.equal(out[0], out[1]), L


@pytest.mark.parametrize("L0", [2, 16, 30, 44, 58, 90])
def test_every_limb_count_of_the_separate_passes(L0):
    """The separate decomposition and CRT read their accumulators in pairs of 16-column loads, the
    second absent at the end of some: limb counts (and with them prime counts) of every remainder, an
    explicit split, one tile and, past 128 primes, several."""
    torch = _torch()
    import polymult
    ensure_library()
    N, s = 512, torch.cuda.current_stream().cuda_stream
    for L in range(L0, L0 + 14):
        W = 32 * L - 13
        q = orc.limbs_of(_q(N, W), L)
        _, a = _operands(torch, N, W, 1, 3 * L, 0)
        _, b = _operands(torch, N, W, 1, 3 * L + 1, 0)
        c = [torch.full((1, N, L), -1, dtype=torch.int32, device="cuda") for _ in range(2)]
        with polymult.Batch([(N, W, q, 1, a.data_ptr(), b.data_ptr(), c[0].data_ptr(), 5)]) as batch:
            assert batch.class_info(0)["gemm"] == "tensor"
            batch.run(s)
            batch.sync()
        with polymult.Multiplier(N, W, q, gemm="plain") as m:
            m.multiply_device(a.data_ptr(), b.data_ptr(), c[1].data_ptr(), 1, s)
            m.sync()
        assert torch.equal(c[0], c[1]), L


# aligned operands (bulk copies) and operands off the 16-byte boundary (plain loads), each form's
# decomposition: with the column stages, in prime blocks, on the CUDA cores
FORMS = [(512, 300, "tensor"), (512, 3000, "tensor"), (512, 300, "plain")]


def _one_by_one(torch, m, a, b, s):
    c = torch.zeros(a.shape, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    m.multiply_device(a.data_ptr(), b.data_ptr(), c.data_ptr(), 1, s)
    m.sync()
    return c


@pytest.mark.parametrize("off", [0, 1])
@pytest.mark.parametrize("N,W,gemm", FORMS)
def test_operands_of_the_kernel_before(N, W, gemm, off):
    """Operands that the kernel before the call has just written, over older ones that calls have just
    read, and products that are the next call's operand: those of calls run one by one."""
    torch = _torch()
    import polymult
    ensure_library()
    L, s = (W + 31) // 32, torch.cuda.current_stream().cuda_stream
    _, xs = _operands(torch, N, W, 5, 8, 0)
    _, b = _operands(torch, N, W, 1, 9, off)
    bufs = torch.zeros((7, N * L + 64), dtype=torch.int32, device="cuda")

    def at(k):
        return bufs[k, off:off + N * L].view(N, L)
    with polymult.Multiplier(N, W, orc.limbs_of(_q(N, W), L), gemm=gemm) as m:
        want = [_one_by_one(torch, m, xs[i].clone(), b[0], s) for i in range(5)]
        chain = want[0]
        for _ in range(5):
            c = torch.zeros(N * L + 1, dtype=torch.int32, device="cuda")[off:off + N * L].view(N, L)
            c.copy_(chain)
            chain = _one_by_one(torch, m, c, b[0], s)
        a, got = at(0), []
        for i in range(5):
            torch.bitwise_or(xs[i], 0, out=a)
            c = torch.zeros((N, L), dtype=torch.int32, device="cuda")
            m.multiply_device(a.data_ptr(), b.data_ptr(), c.data_ptr(), 1, s)
            a.fill_(-1)
            got.append(c)
        torch.bitwise_or(xs[0], 0, out=a)
        for k in range(6):
            m.multiply_device(at(k).data_ptr(), b.data_ptr(), at(k + 1).data_ptr(), 1, s)
        m.sync()
        for g, w in zip(got, want):
            assert torch.equal(g, w)
        assert torch.equal(at(6), chain)


@pytest.mark.parametrize("graph", [None, True, False])
@pytest.mark.parametrize("N,W,gemm", FORMS)
def test_operands_of_another_stream(N, W, gemm, graph):
    """Operands written on another stream and handed over by an event, overwritten there once the call
    is done: a Multiplier's call, and a batch's run, whose streams wait for an event of their own."""
    torch = _torch()
    import polymult
    ensure_library()
    L = (W + 31) // 32
    q = orc.limbs_of(_q(N, W), L)
    _, xs = _operands(torch, N, W, 6, 8, 0)
    _, b = _operands(torch, N, W, 1, 9, 0)
    s1, s2 = torch.cuda.Stream(), torch.cuda.Stream()
    a = torch.zeros((N, L), dtype=torch.int32, device="cuda")
    c = torch.zeros_like(a)
    got = [torch.zeros_like(a) for _ in range(6)]
    with polymult.Multiplier(N, W, q, gemm=gemm) as m:
        want = [_one_by_one(torch, m, xs[i].clone(), b[0], s1.cuda_stream) for i in range(6)]
        batch = None
        if graph is not None:
            batch = polymult.Batch([(N, W, q, 1, a.data_ptr(), b.data_ptr(), c.data_ptr())], gemm=gemm, graph=graph)
        torch.cuda.synchronize()
        written, done = torch.cuda.Event(), torch.cuda.Event()
        for i in range(6):
            with torch.cuda.stream(s2):
                if i:
                    s2.wait_event(done)
                a.fill_(-1)
                torch.bitwise_or(xs[i], 0, out=a)
                written.record(s2)
            s1.wait_event(written)
            if batch is None:
                m.multiply_device(a.data_ptr(), b.data_ptr(), c.data_ptr(), 1, s1.cuda_stream)
            else:
                batch.run(s1.cuda_stream)
            with torch.cuda.stream(s1):
                torch.bitwise_or(c, 0, out=got[i])
                done.record(s1)
        torch.cuda.synchronize()
        if batch is not None:
            batch.sync()
            batch.close()
        m.sync()
    for g, w in zip(got, want):
        assert torch.equal(g, w)


@pytest.mark.parametrize("N,W", [(2048, 64), (4096, 256), (2048, 868), (2048, 1001)])
def test_scratch_of_the_pair_layout(monkeypatch, N, W):
    """Residue scratch: the primes of a multiply, rounded up to an even number, and launch groups that
    stay within POLYMULT_GROUP_WORDS; the last multiplies of a group hold the same products."""
    torch = _torch()
    import polymult
    ensure_library()
    L, count = (W + 31) // 32, 7
    q = orc.limbs_of(_q(N, W), L)
    _, a = _operands(torch, N, W, count, 1, 0)
    _, b = _operands(torch, N, W, count, 2, 0)
    s = torch.cuda.current_stream().cuda_stream
    with polymult.Multiplier(N, W, q, gemm="plain") as m:
        want = torch.zeros_like(a)
        m.multiply_device(a.data_ptr(), b.data_ptr(), want.data_ptr(), count, s)
        m.sync()
        K = m.info()["K"]
    words = 5 * (K + K % 2) * N + 1
    monkeypatch.setenv("POLYMULT_GROUP_WORDS", str(words))
    with polymult.Multiplier(N, W, q) as m:
        assert m.info()["launches_per_multiply"] == 3
        assert m.info()["scratch_bytes"] == 2 * 4 * (K + K % 2) * N
        c = torch.zeros_like(a)
        m.multiply_device(a.data_ptr(), b.data_ptr(), c.data_ptr(), count, s)
        m.sync()
        assert m.info()["group"] == 5 and m.info()["scratch_bytes"] <= 2 * 4 * words
    assert torch.equal(c, want)


@pytest.mark.parametrize("N,W,body", [(512, 300, 16), (1024, 300, 32), (2048, 300, 32), (4096, 300, 64), (8192, 868, 128)])
def test_narrow_host_chunks(N, W, body):
    """The separate passes of an engine whose rows' twiddles lie by thread: host schedules with chunks
    below a tile's 8 columns, at each row length they reach."""
    torch = _torch()
    import polymult
    ensure_library()
    L = (W + 31) // 32
    xa, a = _operands(torch, N, W, 1, 5, 0)
    xb, b = _operands(torch, N, W, 1, 6, 0)
    c = torch.zeros((1, N, L), dtype=torch.int32, device="cuda")
    with polymult.Multiplier(N, W, orc.limbs_of(_q(N, W), L)) as m:
        assert m.info()["launches_per_multiply"] == 3 and N // 16 // body < 8
        m.multiply_device(a.data_ptr(), b.data_ptr(), c.data_ptr(), 1, torch.cuda.current_stream().cuda_stream)
        m.sync()
        m.set_pipeline(body, body)
        got = m.multiply(xa[0], xb[0])
    assert np.array_equal(got, c.cpu().numpy().view(np.uint32)[0])


@pytest.mark.parametrize("N,W", [(512, 64), (4096, 868), (65536, 1747)])
def test_tables_of_the_fused_form(N, W):
    """The fused form's tables beside the separate passes': its constant images, no second copy of the
    twiddles."""
    _torch()
    import polymult
    ensure_library()
    got = []
    for gemm in ("tensor", "plain"):
        with polymult.Multiplier(N, W, orc.limbs_of(_q(N, W), (W + 31) // 32), gemm=gemm) as m:
            got.append(m.info())
    assert got[0]["launches_per_multiply"] == 3
    # 4 constant bytes x at most 256 rows x at most 256 K bytes for each operand, 256 x 512 for the CRT,
    # 15 twiddles, p and floor(2^48 / p) of up to 128 primes
    assert got[0]["table_bytes"] - got[1]["table_bytes"] <= 2 * 4 * 256 * 256 + 256 * 512 + 128 * (15 * 8 + 4)


@pytest.mark.parametrize("N,W", [(512, 64), (4096, 256), (8192, 200), (8192, 250), (4096, 520)])
def test_small_host_calls(N, W):
    """Host calls around the size below which a call runs in one stream (operands of 256 KB), one after
    another, from pageable and page-locked buffers and with one of the three page-locked."""
    torch = _torch()
    import polymult
    ensure_library()
    L = (W + 31) // 32
    xs, ds = _operands(torch, N, W, 4, 11, 0)
    want = torch.zeros((3, N, L), dtype=torch.int32, device="cuda")
    pinned = [torch.from_numpy(x.view(np.int32).copy()).pin_memory().numpy().view(np.uint32) for x in xs]
    with polymult.Multiplier(N, W, orc.limbs_of(_q(N, W), L)) as m:
        for i in range(3):
            m.multiply_device(ds[i].data_ptr(), ds[i + 1].data_ptr(), want[i].data_ptr(), 1,
                              torch.cuda.current_stream().cuda_stream)
        m.sync()
        want = want.cpu().numpy().view(np.uint32)
        for pa, pb, pc in [(0, 0, 0), (1, 1, 1), (1, 0, 0), (0, 1, 0), (0, 0, 1)]:
            for i in range(3):
                out = torch.zeros((N, L), dtype=torch.int32)
                out = (out.pin_memory() if pc else out).numpy().view(np.uint32)
                m.multiply((pinned if pa else xs)[i], (pinned if pb else xs)[i + 1], out=out)
                assert np.array_equal(out, want[i]), (pa, pb, pc, i)
