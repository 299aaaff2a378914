"""GPU: kernels at the sizes where their tiling or the choice between two paths can go wrong.

Bytes are compared exactly with the host mirror of the reference's quantisers (amd_optimization_challenge_b200.inputs);
attention results with the fp32 oracle at the tolerances of tests/helpers.py."""
import pytest
import torch

from helpers import assert_close, oracle_for_data
from oracle import mla_oracle as mo

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def pkg():
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    import amd_optimization_challenge_b200 as pkg
    return pkg


# a block covers 8 rows of an e4m3 cache at a time and 4 of the others; 148 * 7 blocks, the one for the status word among them, are one step of
# the grid (8280 and 4140 rows)
@pytest.mark.parametrize("n", [1, 3, 4, 5, 4143, 4145, 8289])
@pytest.mark.parametrize("listed", [False, True])
def test_append_rows_around_the_steps_of_block_and_grid(pkg, n, listed):
    from amd_optimization_challenge_b200 import inputs
    g = torch.Generator().manual_seed(n)
    kv = torch.randn(n, 1, 576, generator=g).bfloat16()
    kv[:, 0, 7] = -0.0
    kv[n // 2, 0, 64:96] = 0.0
    pool, base = n + 9, 5
    slots = torch.randperm(pool, generator=g)[:n] if listed else base + torch.arange(n)
    where = dict(slots=slots.to(torch.int32).cuda()) if listed else dict(base_slot=base)
    u8 = dict(dtype=torch.uint8, device="cuda")
    c8, s8 = inputs.quantize_fp8(kv)
    c4, s4 = inputs.quantize_mxfp4(kv)
    want8, want4 = c8.view(torch.uint8).reshape(n, 576), c4.reshape(n, 288)
    full = lambda rows, t: torch.full((pool, t.shape[1]), 0xEE, dtype=torch.uint8).index_copy_(0, rows, t)
    got8 = torch.full((pool, 576), 0xEE, **u8)
    assert int(pkg.kv_append(kv.cuda(), "fp8", (got8, s8.cuda()), **where)) == 0
    assert torch.equal(got8.cpu(), full(slots, want8))
    got4, gots = torch.full((pool, 288), 0xEE, **u8), torch.full((pool, 18), 0xEE, **u8)
    assert int(pkg.kv_append(kv.cuda(), "mxfp4", (got4, gots), **where)) == 0
    assert torch.equal(got4.cpu(), full(slots, want4))
    assert torch.equal(gots.cpu(), full(slots, s4[:, :18].contiguous().view(torch.uint8)))
    hyb = torch.full((pool, 256), 0xEE, **u8), torch.full((pool, 16), 0xEE, **u8), torch.full((pool, 64), 0xEE, **u8)
    assert int(pkg.kv_append(kv.cuda(), "hybrid", (*hyb, s8.cuda()), **where)) == 0
    for plane, rows in zip(hyb, (want4[:, :256], s4[:, :16].contiguous().view(torch.uint8), want8[:, 512:])):
        assert torch.equal(plane.cpu(), full(slots, rows.contiguous()))
    if listed:                                                   # a slot outside the pool: its row is dropped, the rest is written
        bad = slots.to(torch.int32)
        bad[n - 1] = pool
        got8.fill_(0xEE)
        assert int(pkg.kv_append(kv.cuda(), "fp8", (got8, s8.cuda()), slots=bad.cuda())) == 1
        assert torch.equal(got8.cpu(), full(slots[:n - 1], want8[:n - 1]))


def test_append_and_merge_behind_other_work_of_the_stream(pkg):
    """Their blocks are placed while the kernel before them drains: what that kernel writes has to be seen, in a graph too."""
    from amd_optimization_challenge_b200 import inputs
    g = torch.Generator().manual_seed(2)
    kv = torch.randn(2000, 1, 576, generator=g).bfloat16()
    codes, scale = inputs.quantize_fp8(kv)
    want = codes.view(torch.uint8).reshape(2000, 576)
    src, dev_scale = kv.cuda(), scale.cuda()
    staged, cache = torch.zeros_like(src), torch.zeros(2000, 576, dtype=torch.uint8, device="cuda")
    big = torch.empty(1 << 26, device="cuda")

    def step():
        big.fill_(1.0)
        staged.copy_(src)
        pkg.kv_append(staged, "fp8", (cache, dev_scale))
        return cache.clone()

    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        first = step()
    torch.cuda.synchronize()
    assert torch.equal(first.cpu(), want)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = step()
    for _ in range(3):
        staged.zero_()
        cache.zero_()
        out.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out.cpu(), want)


@pytest.mark.parametrize("parts", [1, 7, 8, 9, 17])
def test_merge_around_the_group_of_parts_in_flight(pkg, parts):
    """Eight parts are loaded at a time.  fp32 sums of at most 17 terms: the bf16 output is within one rounding."""
    g = torch.Generator().manual_seed(parts)
    o, lse = torch.randn(parts, 5, 3, 512, generator=g), 4 * torch.randn(parts, 5, 3, generator=g)
    lse[parts // 2, 1] = float("-inf")                           # an empty part
    lse[:, 2, 1] = float("-inf")                                 # an empty row
    o[parts // 2, 1] = 0
    w = torch.softmax(lse.double(), 0).nan_to_num(0.0)
    want = (w[..., None] * o.double()).sum(0)
    got, got_lse = pkg.combine_partials(o.cuda(), lse.cuda(), return_lse=True)
    assert torch.allclose(got.cpu().double(), want, rtol=2 ** -8, atol=1e-5)
    assert torch.allclose(got_lse.cpu().double(), torch.logsumexp(lse.double(), 0), atol=1e-5)


def _run(pkg, data, kv_format, q_format, **more):
    cfg = dict(data[4], kv_format=kv_format, q_format=q_format, **more)
    return pkg.custom_kernel((*data[:4], cfg))


# Tiles have 96 tokens (e4m3 cache, up to 32 rows) or 128, units of 16 tokens in two alternating halves; rows select the
# 16, 32 and 64 row kernels and several row groups of the last.
@pytest.mark.parametrize("heads,q_len", [(16, 1), (16, 2), (64, 1), (64, 2)])
@pytest.mark.parametrize("kv_format,q_format", [("fp8", "fp8"), ("fp8", "bf16"), ("mxfp4", "fp8"), ("mxfp4", "bf16"),
                                                ("hybrid", "fp8"), ("hybrid", "bf16")])
def test_lengths_around_units_and_tiles(pkg, kv_format, q_format, heads, q_len):
    lens = [15, 16, 17, 95, 96, 97, 0, 111, 112, 127, 128, 129, 191, 192, 193, 255, 256, 257, 289, 385]
    data = pkg.generate_input(len(lens), q_len, max(lens), seed=heads + q_len, kv_lens=lens, shuffle_pages=True,
                              num_heads=heads, formats=(kv_format,))
    want = oracle_for_data(data, kv_format, q_format)
    for max_ctas in (0, 5):                                      # a tile or less for each CTA; several tiles and sequences
        assert_close(_run(pkg, data, kv_format, q_format, impl="tcgen05", max_ctas=max_ctas), want, tight=1.5e-2)


def _run_over_nans(pkg, data, kv_format, q_format, **more):
    """_run whose output block holds NaNs before the call: a row that nobody writes is seen."""
    block = torch.full((data[0].shape[0], data[0].shape[1], 512), float("nan"), dtype=torch.bfloat16, device="cuda")
    at = block.data_ptr()
    del block
    out = _run(pkg, data, kv_format, q_format, **more)
    assert out.data_ptr() == at
    return out


def _left(pkg):
    """CTAs that have left a meeting of eager calls before all had come (word 4 of the workspaces)."""
    from amd_optimization_challenge_b200 import submission
    return sum(int(ws[16:20].view(torch.int32)) for ws in submission._workspace_cache.values())


# CTAs that do not wait for one another (0 cycles), or not for long: they look at the shares of Q that nobody has looked at, and those
# that are late merge what the others had to leave behind.
@pytest.mark.parametrize("kv_format,q_format,heads,lens", [("fp8", "fp8", 16, [900, 0, 97, 2000]), ("mxfp4", "bf16", 32, [4000]),
                                                           ("hybrid", "fp8", 128, [700, 1500, 64]), ("fp8", "bf16", 16, [130] * 300),
                                                           ("fp8", "fp8", 128, [3] * 150 + [6000, 0, 9000] + [3] * 150)])
def test_ctas_that_leave_before_the_merge(pkg, monkeypatch, kv_format, q_format, heads, lens):
    data = pkg.generate_input(len(lens), 1, max(lens), seed=heads, kv_lens=lens, shuffle_pages=True, num_heads=heads, formats=(kv_format,))
    want = _run(pkg, data, kv_format, q_format, impl="tcgen05")
    assert torch.isfinite(want).all()
    for cycles in (0, 300, 0, 1000, 2000, 4000, 6000, 8000, 12000, 20000, 0):     # up to the time that they are apart
        monkeypatch.setenv("B200_MLA_MEET_CYCLES", str(cycles))
        before = _left(pkg)
        for _ in range(5):
            assert torch.equal(_run_over_nans(pkg, data, kv_format, q_format, impl="tcgen05"), want)
        assert cycles or _left(pkg) > before
    monkeypatch.delenv("B200_MLA_MEET_CYCLES")
    # and the words they meet at are zero afterwards
    assert torch.equal(_run_over_nans(pkg, data, kv_format, q_format, impl="tcgen05", check_status=True), want)


@pytest.mark.parametrize("text", ["", "soon", "-1", "0x", "0 us", "+0", " 0", "99999999999999999999"])
def test_a_limit_that_is_no_number_is_ignored(pkg, monkeypatch, text):
    data = pkg.generate_input(4, 1, 900, seed=4, kv_lens=[900] * 4)
    _run(pkg, data, "fp8", "fp8", impl="tcgen05")
    before = _left(pkg)
    monkeypatch.setenv("B200_MLA_MEET_CYCLES", text)
    for _ in range(5):
        _run(pkg, data, "fp8", "fp8", impl="tcgen05")
    assert _left(pkg) == before


# What CTAs leave behind must not all fall on one of them, and no CTA has to look at all of a large Q: these calls took ten times as
# long when they did.
@pytest.mark.parametrize("kv_format,q_format,lens", [("fp8", "bf16", [3000] * 24), ("fp8", "fp8", [100] * 600)])
def test_a_call_whose_ctas_leave_takes_little_longer(pkg, monkeypatch, kv_format, q_format, lens):
    data = pkg.generate_input(len(lens), 1, max(lens), seed=3, kv_lens=lens, num_heads=128, formats=(kv_format,))

    def us(n=20):
        times = []
        for _ in range(5):
            start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            torch.cuda._sleep(2_000_000)
            start.record()
            for _ in range(n):
                _run(pkg, data, kv_format, q_format)
            end.record()
            torch.cuda.synchronize()
            times.append(start.elapsed_time(end) * 1e3 / n)
        return min(times)

    waiting = us()
    monkeypatch.setenv("B200_MLA_MEET_CYCLES", "0")
    leaving = us()
    assert leaving <= 3 * waiting, f"{leaving:.0f} us, {waiting:.0f} us where CTAs wait"


@pytest.mark.parametrize("kv_format,q_format", [("fp8", "fp8"), ("mxfp4", "bf16")])
def test_decode_behind_other_work_of_the_stream(pkg, kv_format, q_format):
    """Its CTAs are placed while the kernel before them drains: what that kernel writes has to be seen, in a graph too."""
    lens = [3000, 17, 900, 64]
    sets = [pkg.generate_input(4, 1, 3000, seed=s, kv_lens=lens, shuffle_pages=True, formats=(kv_format,)) for s in (1, 2)]
    want = [_run(pkg, d, kv_format, q_format) for d in sets]
    torch.cuda.synchronize()
    q, planes, table = sets[0][0].clone(), tuple(t.clone() for t in sets[0][1][kv_format]), sets[0][4]["kv_indices"].clone()
    data = (q, {kv_format: planes}, *sets[0][2:4], dict(sets[0][4], kv_indices=table))

    def step(i):
        for to, new in zip(planes, sets[i][1][kv_format]):
            to.view(torch.uint8).copy_(new.view(torch.uint8))
        table.copy_(sets[i][4]["kv_indices"])
        q.copy_(sets[i][0])
        return _run(pkg, data, kv_format, q_format)

    outs = [step(i & 1) for i in range(10)]
    assert all(torch.equal(o, want[i & 1]) for i, o in enumerate(outs))
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        outs = [step(i & 1) for i in range(4)]
    for _ in range(3):
        graph.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(o, want[i & 1]) for i, o in enumerate(outs))


def _eager_and_captured(steps, want, rounds=3):
    """Every step's output, eagerly one after the other and as a graph."""
    outs = [step() for _ in range(rounds) for step in steps]
    for i, o in enumerate(outs):
        assert torch.equal(o, want[i % len(want)]), i
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        outs = [step() for step in steps]
    for _ in range(rounds):
        graph.replay()
        torch.cuda.synchronize()
        for i, o in enumerate(outs):
            assert torch.equal(o, want[i]), i


# Only the edge between two kernels is relaxed (a copy before the decode orders it fully): here a kernel has written each of the
# inputs in turn just before the decode, with inputs that change from call to call.
@pytest.mark.parametrize("kv_format,q_format", [("fp8", "fp8"), ("fp8", "bf16"), ("mxfp4", "bf16"), ("hybrid", "fp8")])
def test_decode_behind_the_kernel_that_wrote_an_input(pkg, kv_format, q_format):
    lens = ([3000, 17, 900, 64], [64, 900, 17, 3000])
    sets = [pkg.generate_input(4, 1, 3000, seed=s, kv_lens=l, shuffle_pages=True, formats=(kv_format,)) for s, l in zip((1, 2), lens)]
    want = [_run(pkg, d, kv_format, q_format) for d in sets]
    assert not torch.equal(*want)
    inputs = [(d[0], d[3], d[4]["kv_indices"], *d[1][kv_format]) for d in sets]
    own = [t.clone() for t in inputs[0]]
    data = (own[0], {kv_format: tuple(own[3:])}, sets[0][2], own[1], dict(sets[0][4], kv_indices=own[2]))

    def write(to, new):
        if to.dtype in (torch.bfloat16, torch.float32):
            torch.maximum(new, new, out=to)
        else:                                                    # indices, and bytes of every kind
            kind = torch.int32 if to.dtype is torch.int32 else torch.uint8
            torch.bitwise_or(new.view(kind), new.view(kind), out=to.view(kind))

    def step(i, last):
        order = [k for k in range(len(own)) if k != last] + [last]
        for k in order:
            write(own[k], inputs[i][k])
        return _run(pkg, data, kv_format, q_format)

    todo = [(n & 1, n % len(own)) for n in range(2 * len(own))] + [(n + 1 & 1, n % len(own)) for n in range(2 * len(own))]
    torch.cuda.synchronize()
    _eager_and_captured([lambda i=i, last=last: step(i, last) for i, last in todo], [want[i] for i, _ in todo])


# The same behind the library's own kernels: rows appended, Q quantised, and partials that a merge still reads.
@pytest.mark.parametrize("kv_format", ["fp8", "mxfp4", "hybrid"])
def test_decode_behind_kernels_of_the_library(pkg, kv_format):
    lens = [3000, 17, 900, 64]
    n, heads = sum(lens), 16
    g = torch.Generator(device="cuda").manual_seed(5)
    rows = [torch.randn(n, 576, generator=g, device="cuda").bfloat16() for _ in range(2)]
    qs = [torch.randn(4, heads, 576, generator=g, device="cuda").bfloat16() for _ in range(2)]
    slots = torch.randperm(n, generator=g, device="cuda").to(torch.int32)
    planes = {"fp8": pkg.quantize_fp8, "mxfp4": pkg.quantize_mxfp4, "hybrid": pkg.quantize_hybrid}[kv_format](rows[0][:, None])
    planes = tuple(t.clone() for t in planes)
    ip = torch.tensor([0, 3000, 3017, 3917, 3981], dtype=torch.int32, device="cuda")
    n_o = 4 * heads * 512
    record = torch.empty(2 * (n_o + 4 * heads), device="cuda")
    parts = [(r[:n_o].view(4, heads, 512), r[n_o:].view(4, heads)) for r in record.chunk(2)]

    def step(i, last, wait):
        pause = torch.cuda.synchronize if wait else lambda: None
        if last == "append":
            q, scale = pkg.quantize_q_fp8(qs[i])
            pause()
        pkg.kv_append(rows[i], kv_format, planes, slots=slots)
        pause()
        if last == "quantise":
            q, scale = pkg.quantize_q_fp8(qs[i])
            pause()
        for part in parts:
            pkg.mla_decode(q, scale, kv_format, planes, ip, sm_scale=0.05, kv_indices=slots, return_partial=True, partial_out=part)
            pause()
        out = pkg.submission.combine_partials_strided(record, 2, record.numel() // 2, n_o, 4, heads)
        pause()
        return out

    todo = [(k & 1, last) for k in range(4) for last in ("append", "quantise")] + [(k + 1 & 1, last) for k in range(4) for last in ("quantise", "append")]
    want = [step(i, last, True) for i, last in todo]
    assert not torch.equal(want[0], want[2])
    _eager_and_captured([lambda i=i, last=last: step(i, last, False) for i, last in todo], want)


# The span search gives a lane ceil(batch / 32) sequences and looks inside them 32 at a time.
@pytest.mark.parametrize("batch", [31, 32, 33, 64, 65, 300, 1025])
def test_batches_around_the_lanes_of_the_span_search(pkg, batch):
    g = torch.Generator().manual_seed(batch)
    lens = torch.randint(0, 200, (batch,), generator=g).tolist()
    data = pkg.generate_input(batch, 1, 200, seed=batch, kv_lens=lens, formats=("fp8",))
    for max_ctas in (0, 2):
        got = _run(pkg, data, "fp8", "fp8", impl="tcgen05", max_ctas=max_ctas)
        assert_close(got, _run(pkg, data, "fp8", "fp8", impl="generic"), tight=1.5e-2)


# 16 rows of an e4m3 cache come as one box where a page holds them side by side, else row by row; block-scaled units keep
# the page ids of their 16 tokens; sizes that are no power of two divide.
@pytest.mark.parametrize("page", [2, 15, 16, 24, 48, 64, 128])
@pytest.mark.parametrize("kv_format", ["fp8", "mxfp4", "hybrid"])
def test_page_sizes(pkg, kv_format, page):
    from oracle import mla_oracle as mo
    g = torch.Generator().manual_seed(page)
    lens = [1, 200, page, 0, 3 * page + 1, 500]
    per = [(n + page - 1) // page for n in lens]
    npages = sum(per) + 3
    q, kvd, _, _, cfg = pkg.generate_input(len(lens), 1, 500, seed=page, kv_lens=[npages * page] + [0] * 5, formats=(kv_format,))
    ids = torch.randperm(npages, generator=g)[:sum(per)].to(torch.int32)
    cum = lambda v: torch.tensor([0] + v, dtype=torch.int32).cumsum(0).to(torch.int32)
    page_indptr, ip = cum(per), cum(lens)
    got = pkg.mla_decode(q, None, kv_format, kvd[kv_format], ip.cuda(), sm_scale=cfg["sm_scale"], kv_indices=ids.cuda(),
                         page_size=page, kv_page_indptr=page_indptr.cuda(), impl="tcgen05")
    slots = [int(ids[page_indptr[b] + t // page]) * page + t % page for b, n in enumerate(lens) for t in range(n)]
    want = mo.decode_from_data(q.cpu(), None, kv_format, tuple(t.cpu() for t in kvd[kv_format]), ip.numpy(),
                               torch.tensor(slots, dtype=torch.int32).numpy(), cfg["sm_scale"])
    assert_close(got, want, tight=1.5e-2)


@pytest.mark.parametrize("kv_format", ["fp8", "mxfp4", "hybrid"])
@pytest.mark.parametrize("heads,batch", [(16, 1), (32, 7), (128, 3)])
def test_q_quantised_in_the_call_equals_two_steps(pkg, kv_format, heads, batch):
    """One launch finds the maximum of Q across its CTAs: the bits of quantize_q_fp8 and a decode of its codes."""
    lens = [700 - 97 * i for i in range(batch)]
    data = pkg.generate_input(batch, 1, 700, seed=batch, kv_lens=lens, num_heads=heads, formats=(kv_format,))
    q, kvd, _, ip, cfg = data
    q[-1, -1, 575] = -9.0                                        # the maximum is in the last element
    codes, scale = pkg.quantize_q_fp8(q)
    two = pkg.mla_decode(codes, scale, kv_format, kvd[kv_format], ip, sm_scale=cfg["sm_scale"], impl="tcgen05")
    for _ in range(3):                                           # the words the CTAs met at are zero again after every call
        assert torch.equal(_run(pkg, data, kv_format, "fp8", impl="tcgen05"), two)


def test_repeated_calls_notice_what_changes(pkg):
    """Repeated calls of the same objects go through a kept plan; new values, lengths, tensors and streams must count."""
    data = pkg.generate_input(3, 1, 300, seed=3, kv_lens=[300, 40, 7], shuffle_pages=True, formats=("fp8",))
    data = (*data[:4], dict(data[4], kv_format="fp8", q_format="fp8"))
    check = lambda d: assert_close(pkg.custom_kernel(d), oracle_for_data(d, "fp8", "fp8"), tight=1.5e-2)
    for _ in range(3):
        check(data)
    data[0].mul_(-0.5)                                           # same tensor, other values
    check(data)
    data[3].copy_(torch.tensor([0, 200, 201, 300], dtype=torch.int32))
    check(data)
    other = (data[0].flip(1).contiguous(), *data[1:])            # another Q
    check(other)
    data[4]["sm_scale"] *= 0.5                                   # the configuration in place
    check(data)
    data[1]["fp8"] = (data[1]["fp8"][0].flip(0).contiguous(), data[1]["fp8"][1])
    check(data)


def test_two_streams_and_threads_with_one_shape(pkg):
    """Scratch belongs to a stream: the same shape in two streams, from two threads, at the same time."""
    import threading
    lens = [3000, 17, 900]
    sets = [pkg.generate_input(3, 1, 3000, seed=s, kv_lens=lens, shuffle_pages=True, formats=("fp8",)) for s in (1, 2)]
    sets = [(*d[:4], dict(d[4], kv_format="fp8", q_format="fp8")) for d in sets]
    want = [pkg.custom_kernel(d) for d in sets]
    torch.cuda.synchronize()
    bad = []

    def worker(i):
        with torch.cuda.stream(torch.cuda.Stream()):
            outs = [pkg.custom_kernel(sets[i]) for _ in range(50)]
            torch.cuda.current_stream().synchronize()
        bad.extend(1 for o in outs if not torch.equal(o, want[i]))

    threads = [threading.Thread(target=worker, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad


# Keys `depth` binades below a dominant one, all alike, so that the rounding of their probabilities does not average out.  A
# stored probability ends 2^-17 below the reference maximum (half of that is the largest error), the output is bf16.
@pytest.mark.parametrize("heads", [16, 32, 64, 128])
@pytest.mark.parametrize("depth", [10, 12, 15])
@pytest.mark.parametrize("at", [0, 3000])
def test_coherent_tail_far_below_the_maximum(pkg, heads, depth, at):
    n = 4097
    g = torch.Generator().manual_seed(depth)
    q = torch.zeros(1, heads, 576)
    q[..., 0] = 4.0
    kv = 1.0 + 0.25 * torch.randn(n, 576, generator=g)
    kv[:, 0], kv[:, 512:] = 0.0, 0.0
    kv[at, 0], kv[at, 1:512] = depth * 0.6931 / 4.0, 0.1 * torch.randn(511, generator=g)
    codes, scale = pkg.quantize_fp8(kv.bfloat16().cuda())
    qc, qs = pkg.quantize_q_fp8(q.bfloat16().cuda())
    K = codes.reshape(n, 576).float().double() * scale.double()
    want = torch.softmax(qc[0].float().double() * qs.double() @ K.T, -1) @ K[:, :512]
    ip = torch.tensor([0, n], dtype=torch.int32, device="cuda")
    for max_ctas in (1, 0):
        got = pkg.mla_decode(qc, qs, "fp8", (codes, scale), ip, sm_scale=1.0, impl="tcgen05", max_ctas=max_ctas)[0].double()
        assert float((got - want).norm() / want.norm()) <= 2.0 ** (depth - 18) + 2.0 ** -8


# Scores that climb along the sequence, for different rows at different tiles, so that reference maxima move and O is rescaled
# again and again.  Against the fp32 oracle: a bf16 output (2^-9), probabilities of about eight bits (2^-9), Q and cache as they are
# stored; with as much again for their sum.
@pytest.mark.parametrize("kv_format,q_format,heads", [("fp8", "fp8", 16), ("fp8", "bf16", 32), ("fp8", "fp8", 64), ("fp8", "fp8", 128),
                                                      ("mxfp4", "bf16", 16), ("mxfp4", "bf16", 32), ("mxfp4", "fp8", 64), ("hybrid", "fp8", 128)])
def test_reference_maxima_that_move_at_most_tiles(pkg, kv_format, q_format, heads):
    lens, g = [1500, 97, 700], torch.Generator().manual_seed(heads)
    n = sum(lens)
    kv = 0.5 * torch.randn(n, 1, 576, generator=g)
    at = torch.cat([torch.arange(k) for k in lens]).float()
    for j in range(4):
        kv[:, 0, 32 * j] = at * (0.5 + j) / 700
    q = 0.2 * torch.randn(3, heads, 576, generator=g)
    for h in range(heads):
        q[:, h, 32 * (h % 4)] = 4.0
    quantise = {"fp8": pkg.quantize_fp8, "mxfp4": pkg.quantize_mxfp4, "hybrid": pkg.quantize_hybrid}[kv_format]
    planes, q = quantise(kv.bfloat16().cuda()), q.bfloat16().cuda()
    qc, qs = pkg.quantize_q_fp8(q) if q_format == "fp8" else (q, None)
    ip = torch.tensor([0, 1500, 1597, 2297], dtype=torch.int32, device="cuda")
    run = lambda **kw: pkg.mla_decode(qc, qs, kv_format, planes, ip, sm_scale=1.0, **kw).float().cpu()
    want = mo.decode_from_data(qc.cpu(), None if qs is None else qs.cpu(), kv_format, tuple(t.cpu() for t in planes), ip.cpu().numpy(), None,
                               1.0).float()
    for kw in (dict(impl="generic"), dict(impl="tcgen05", max_ctas=1), dict(impl="tcgen05")):      # one CTA per row group, and spread out
        got = run(**kw).reshape(want.shape)
        assert torch.isfinite(got).all()
        assert float((got - want).norm() / want.norm()) <= 2.0 ** -7


# The first tiles' scores lie 2^jump below the later ones': a tile whose maximum is far above the reference is read again, so that its
# scores keep their last bits.  They agree with 64 bits to some 1e-6; half an ulp of 256, up to which a tile is shifted instead, is 8e-6
# (5e-6 of the LSE).
@pytest.mark.parametrize("kv_format,q_format,heads,jump", [
    (*kind, jump) for kind in (("fp8", "bf16", 16), ("fp8", "fp8", 16), ("fp8", "fp8", 64), ("mxfp4", "bf16", 16), ("mxfp4", "bf16", 32),
                               ("mxfp4", "fp8", 64), ("hybrid", "fp8", 64))
    for jump in (5, 9, 13, 15, 17, 21) if jump <= 15 or kind[0] != "fp8"])       # an e4m3 cache has one scale: the others would be zeros
def test_a_maximum_that_moves_far(pkg, kv_format, q_format, heads, jump):
    n, g = 2000, torch.Generator().manual_seed(jump)
    kv = torch.randn(n, 1, 576, generator=g)
    kv[:, 0, :32] = 0.0
    kv[:512, 0, :32] = -2.0 ** (jump - 1)
    q = torch.randn(1, heads, 576, generator=g)
    q[..., :32] = 1.0
    planes, q = {"fp8": pkg.quantize_fp8, "mxfp4": pkg.quantize_mxfp4, "hybrid": pkg.quantize_hybrid}[kv_format](kv.bfloat16().cuda()), q.bfloat16().cuda()
    qc, qs = pkg.quantize_q_fp8(q) if q_format == "fp8" else (q, None)
    keys = mo.dequant_kv(kv_format, tuple(t.cpu() for t in planes)).double().reshape(n, 576)
    rows = mo.dequant_q(qc.cpu(), None if qs is None else qs.cpu()).double().reshape(heads, 576)
    scores = rows @ keys.T * 0.0625
    ip = torch.tensor([0, n], dtype=torch.int32, device="cuda")
    o, lse = pkg.mla_decode(qc, qs, kv_format, planes, ip, sm_scale=0.0625, return_partial=True, impl="tcgen05", max_ctas=1)
    assert float((lse.cpu().double().reshape(-1) - torch.logsumexp(scores, 1)).abs().max()) <= 1e-5
    if kv_format == "fp8":
        want = torch.softmax(scores, 1) @ keys[:, :512]
        assert float((o.cpu().double().reshape(heads, 512) - want).norm() / want.norm()) <= 2.0 ** -10


def _captured(pkg, data, n=1, stream=None):
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        outs = [pkg.custom_kernel(data) for _ in range(n)]
    return graph, outs


@pytest.mark.parametrize("kv_format,q_format,heads", [("fp8", "fp8", 16), ("mxfp4", "bf16", 32), ("hybrid", "fp8", 64)])
def test_captures_with_and_without_an_earlier_call(pkg, kv_format, q_format, heads):
    """A graph's scratch is its own: the second capture is replayed first, calls on the capturing stream come in between."""
    lens = [700, 33, 1900, 0, 260]                               # a shape that no other test uses: no scratch from an earlier call
    data = pkg.generate_input(5, 1, 1900, seed=heads, kv_lens=lens, shuffle_pages=True, num_heads=heads, formats=(kv_format,))
    data = (*data[:4], dict(data[4], kv_format=kv_format, q_format=q_format))
    want = oracle_for_data(data, kv_format, q_format)
    s = torch.cuda.Stream()
    g1, o1 = _captured(pkg, data, 2, s)
    g2, o2 = _captured(pkg, data, 1, s)
    with torch.cuda.stream(s):
        for _ in range(2):
            g2.replay()
            assert_close(o2[0], want, tight=1.5e-2)
            eager = pkg.custom_kernel(data)
            assert_close(eager, want, tight=1.5e-2)
        g3, o3 = _captured(pkg, data, 1, s)
        del g2
        for g, o in ((g3, o3), (g1, o1), (g3, o3)):
            [t.zero_() for t in o]
            g.replay()
            assert all(torch.equal(t, eager) for t in o)
    from amd_optimization_challenge_b200 import submission
    assert not submission._graph_pinned                          # the scratch came from the graphs' own pool


def test_replays_beside_calls_and_other_graphs_of_one_shape(pkg):
    lens = [3000, 17, 900, 64]
    sets = [pkg.generate_input(4, 1, 3000, seed=s, kv_lens=lens, shuffle_pages=True, formats=("fp8",)) for s in range(3)]
    sets = [(*d[:4], dict(d[4], kv_format="fp8", q_format="fp8")) for d in sets]
    want = [pkg.custom_kernel(d) for d in sets]
    graphs = [_captured(pkg, d, 20) for d in sets[:2]]
    streams = [torch.cuda.Stream() for _ in sets]
    torch.cuda.synchronize()
    eager = []
    for _ in range(5):
        for (g, _outs), s in zip(graphs, streams):
            with torch.cuda.stream(s):
                g.replay()
        with torch.cuda.stream(streams[2]):
            eager += [pkg.custom_kernel(sets[2]) for _ in range(20)]
    torch.cuda.synchronize()
    for (_g, outs), w in zip(graphs, want):
        assert all(torch.equal(t, w) for t in outs)
    assert all(torch.equal(t, want[2]) for t in eager)


def test_status_of_replays_reaches_read_status(pkg):
    from amd_optimization_challenge_b200 import _cabi, submission
    lens = [40, 41, 42, 43, 44, 45]                              # this test's own shape: its status word is sticky
    data = pkg.generate_input(6, 2, 45, seed=1, kv_lens=lens, shuffle_pages=True, formats=("mxfp4",))
    data = (*data[:4], dict(data[4], kv_format="mxfp4", q_format="bf16"))
    graph, outs = _captured(pkg, data)
    graph.replay()
    assert submission.read_status(outs[0].device, 6, 16, 2) == 0
    data[4]["kv_indices"][100] = 1 << 20                         # outside the cache: reported, read as another row
    graph.replay()
    data[4]["kv_indices"][100] = 0
    graph.replay()
    assert submission.read_status(outs[0].device, 6, 16, 2) == _cabi.STATUS_BAD_PAGE
    assert submission.read_status(outs[0].device, 6, 16, 1) == 0


@pytest.mark.parametrize("what", ["q", "plane", "scales", "kv_indptr", "kv_indices", "num_slots"])
def test_repeated_calls_notice_tensors_changed_in_place(pkg, what):
    """The same objects with other storage, sizes or strides.  (The old storage stays alive here.)"""
    lens = [300, 40, 7]
    data = pkg.generate_input(3, 1, 300, seed=3, kv_lens=lens, shuffle_pages=True, formats=("mxfp4",))
    data = (*data[:4], dict(data[4], kv_format="mxfp4", q_format="bf16"))
    other = pkg.generate_input(3, 1, 300, seed=4, kv_lens=lens, shuffle_pages=True, formats=("mxfp4",))
    (codes, scales), table = data[1]["mxfp4"], data[4]["kv_indices"]
    direct = lambda: pkg.mla_decode(data[0], None, "mxfp4", (codes, scales), data[3], sm_scale=data[4]["sm_scale"], kv_indices=table,
                                    total_kv_hint=sum(lens))
    check = lambda: [assert_close(o, oracle_for_data(data, "mxfp4", "bf16"), tight=1.5e-2) for o in (pkg.custom_kernel(data), direct())]
    for _ in range(2):
        check()
    keep = [t.clone() for t in (data[0], codes, scales, data[3], table)], [t.detach() for t in (data[0], codes, scales, data[3], table)]
    if what == "q":
        data[0].data = other[0]
    elif what == "plane":
        codes.data = other[1]["mxfp4"][0]
    elif what == "scales":                                       # the same rows behind another stride
        wide = torch.zeros(scales.shape[0], 64, dtype=torch.uint8, device="cuda")
        wide[:, :18] = scales[:, :18]
        scales.data = wide
    elif what == "kv_indptr":
        data[3].data = torch.tensor([0, 200, 201, 300], dtype=torch.int32, device="cuda")
    elif what == "kv_indices":
        table.data = other[4]["kv_indices"]
    else:                                                        # fewer rows at the same address: ids beyond them are not read
        n = codes.shape[0] - 8
        inside = table.clamp(max=n - 1)
        codes.data = codes[:n]
        rows = table.clone()
        assert int((rows >= n).sum()) > 0
        out = pkg.custom_kernel(data)
        table.copy_(inside)
        assert torch.equal(out, pkg.custom_kernel(data))         # read as the last row
        from amd_optimization_challenge_b200 import _cabi, submission
        assert submission.read_status(out.device, 3, 16, 1) == _cabi.STATUS_BAD_PAGE
        ws = submission._workspace(out.device, 3, 16, 1)
        _cabi.check(_cabi.lib.b200_mla_reset_status(ws.data_ptr(), torch.cuda.current_stream().cuda_stream), "reset")
        return
    for _ in range(2):
        check()
    del keep


def test_append_notices_planes_changed_in_place(pkg):
    g = torch.Generator().manual_seed(8)
    rows, scale = torch.randn(40, 576, generator=g).bfloat16().cuda(), torch.full((1,), 0.01, device="cuda")
    store = torch.zeros(100, 576, dtype=torch.uint8, device="cuda")
    plane = store[:50]
    for _ in range(2):
        pkg.kv_append(rows, "fp8", (plane, scale))
    want = store[:40].clone()
    store.zero_()
    plane.as_strided_((50, 576), (1152, 1))                      # every other row of the same memory
    assert int(pkg.kv_append(rows, "fp8", (plane, scale))) == 0
    assert torch.equal(store[:80:2], want) and int(store[1::2].max()) == 0
    plane.as_strided_((39, 576), (1152, 1))                      # a row too few
    with pytest.raises(RuntimeError, match="do not fit"):
        pkg.kv_append(rows, "fp8", (plane, scale))


@pytest.mark.parametrize("kv_format", ["fp8", "mxfp4", "hybrid"])
def test_append_to_planes_with_gaps_between_pages(pkg, kv_format):
    """Rows that no single stride describes, again and again: they reach the planes, and nothing else is written."""
    from amd_optimization_challenge_b200 import inputs
    g = torch.Generator().manual_seed(3)
    pages, used, room = 5, 24, 32
    rows = torch.randn(pages * used, 1, 576, generator=g).bfloat16()
    quant = {"fp8": inputs.quantize_fp8, "mxfp4": inputs.quantize_mxfp4, "hybrid": inputs.quantize_hybrid}[kv_format](rows)
    want = [t.view(torch.uint8).reshape(pages * used, -1) for t in quant if t.dim() > 1]
    gapped = lambda w: torch.full((pages, room, w.shape[1]), 0xEE, dtype=torch.uint8, device="cuda")
    kv, stores = [], []
    for t in quant:
        if t.dim() <= 1:
            kv.append(t.cuda())
        elif t is quant[1]:                                      # E8M0 rows: two-dimensional by contract
            kv.append(torch.full((pages * used, t.shape[-1]), 0xEE, dtype=torch.uint8, device="cuda"))
        else:
            stores.append(gapped(t.view(torch.uint8).reshape(pages * used, -1)))
            kv.append(stores[-1][:, :used])
    for _ in range(3):
        for t in kv:
            if t.dtype == torch.uint8:
                t.fill_(0xEE)
        other = [torch.zeros_like(s) for s in stores]            # takes the place of freed copies
        assert int(pkg.kv_append(rows.cuda(), kv_format, tuple(kv))) == 0
        got = [t.reshape(pages * used, -1).cpu() for t in kv if t.dtype == torch.uint8]
        assert all(torch.equal(a, b) for a, b in zip(got, want))
        assert all(bool((s[:, used:] == 0xEE).all()) for s in stores) and not any(bool(t.any()) for t in other)


@pytest.mark.parametrize("q_format", ["fp8", "bf16"])
@pytest.mark.parametrize("impl", ["tcgen05", "generic"])
def test_one_query_row_that_is_a_slice(pkg, impl, q_format):
    """One query token, its heads a slice of more: contiguous to torch, with the stride of the wider tensor."""
    data = pkg.generate_input(1, 1, 300, seed=6, formats=("fp8",))
    wide = torch.cat((data[0], 3 * data[0], data[0][:, :5]), 1)
    part = (wide[:, :16], *data[1:])
    assert part[0].is_contiguous() and part[0].stride(0) == 37 * 576
    want = oracle_for_data(data, "fp8", q_format)
    for _ in range(2):
        assert_close(_run(pkg, part, "fp8", q_format, impl=impl), want, tight=1.5e-2)


# Special values next to ordinary ones, in both vectors of a thread, and scales at which quotients overflow: the codes of the
# division by the scale.
@pytest.mark.parametrize("scale", [0.01, 1.0, 2.0 ** -100, 2.0 ** 100])
def test_append_casts_special_values_as_the_division_does(pkg, scale):
    g = torch.Generator().manual_seed(1)
    rows = (torch.randn(37, 576, generator=g) * torch.exp2(torch.randint(-40, 40, (37, 576), generator=g).float())).bfloat16()
    rows[3, 8], rows[4, 15], rows[5, 16] = float("inf"), float("-inf"), 3.0e38
    rows[6, 1], rows[7, 9], rows[8, 575] = -3.0e38, float("nan"), -0.0
    q = (rows.float() / torch.tensor(scale)).bfloat16().float()
    want = q.clamp(-448.0, 448.0).to(torch.float8_e4m3fn).view(torch.uint8)
    got = torch.zeros(37, 576, dtype=torch.uint8, device="cuda")
    assert int(pkg.kv_append(rows.cuda(), "fp8", (got, torch.tensor([scale]).cuda()))) == 0
    got, nan = got.cpu(), torch.isnan(q)
    assert torch.equal(got[~nan], want[~nan]) and bool(((got[nan] & 0x7f) == 0x7f).all())


# The same where rows are fetched a step ahead: listed, beyond 5920 of them, 4728 a step of the grid; special rows in each of three
# steps, and a slot list that begins on and off a 16-byte boundary.
@pytest.mark.parametrize("scale,off", [(0.01, 0), (1.0, 3), (2.0 ** -100, 1), (2.0 ** 100, 2)])
def test_append_of_listed_rows_casts_special_values_in_every_step(pkg, scale, off):
    n, pool, g = 9500, 9600, torch.Generator().manual_seed(off)
    rows = (torch.randn(n, 576, generator=g) * torch.exp2(torch.randint(-40, 40, (n, 576), generator=g).float())).bfloat16()
    for r in (0, 4728, 9456):
        rows[r + 3, 8], rows[r + 4, 15], rows[r + 5, 16] = float("inf"), float("-inf"), 3.0e38
        rows[r + 6, 1], rows[r + 7, 9], rows[r + 8, 575] = -3.0e38, float("nan"), -0.0
    q = (rows.float() / torch.tensor(scale)).bfloat16().float()
    want = q.clamp(-448.0, 448.0).to(torch.float8_e4m3fn).view(torch.uint8)
    slots = torch.randperm(pool, generator=g)[:n]
    around = torch.full((n + 8,), -7, dtype=torch.int32, device="cuda")
    listed = around[off:off + n]
    listed.copy_(slots)
    plane = torch.full((pool, 576), 0xEE, dtype=torch.uint8, device="cuda")
    assert int(pkg.kv_append(rows.cuda(), "fp8", (plane, torch.tensor([scale]).cuda()), slots=listed)) == 0
    plane, nan = plane.cpu(), torch.isnan(q)
    got = plane[slots]
    assert torch.equal(got[~nan], want[~nan]) and bool(((got[nan] & 0x7f) == 0x7f).all())
    plane[slots] = 0xEE
    assert bool((plane == 0xEE).all())


# Steps of e4m3 rows are 8 a block, of the others 4.  1035 blocks stay for up to eight steps, then there are 4144; listed e4m3 rows have 591 at any
# of these sizes.
@pytest.mark.parametrize("kv_format,n", [("fp8", 8 * 8288 - 1), ("fp8", 8 * 8288 + 1), ("mxfp4", 4 * 8288 + 1), ("hybrid", 4 * 8288 + 1), ("fp8", 200001)])
def test_append_rows_around_the_wave_rule(pkg, kv_format, n):
    from amd_optimization_challenge_b200 import inputs
    few = torch.randn(997, 1, 576, generator=torch.Generator().manual_seed(n)).bfloat16()
    quant = {"fp8": inputs.quantize_fp8, "mxfp4": inputs.quantize_mxfp4, "hybrid": inputs.quantize_hybrid}[kv_format](few)
    pick = torch.arange(n, device="cuda") % 997
    rows = few.cuda()[pick]
    for slots in (None, torch.randperm(n, device="cuda").to(torch.int32)):
        kv = tuple(torch.zeros(n, t.view(torch.uint8).reshape(997, -1).shape[1], dtype=torch.uint8, device="cuda") if t.dim() > 1 else t.cuda() for t in quant)
        assert int(pkg.kv_append(rows, kv_format, kv, slots=slots)) == 0
        at = slice(None) if slots is None else slots.long()
        for plane, t in zip(kv, quant):
            if t.dim() > 1:
                assert torch.equal(plane[at], t.view(torch.uint8).reshape(997, -1).cuda()[pick])


@pytest.mark.parametrize("off", [0, 1, 2, 3])
@pytest.mark.parametrize("n", [1, 2, 3, 5, 9, 1163])
def test_append_reports_a_bad_slot_wherever_it_stands(pkg, n, off):
    """The slots are looked over one by one up to a 16-byte boundary, then in fours, then one by one."""
    rows = torch.zeros(n, 576, dtype=torch.bfloat16, device="cuda")
    planes = torch.zeros(n, 288, dtype=torch.uint8, device="cuda"), torch.zeros(n, 18, dtype=torch.uint8, device="cuda")
    around = torch.full((n + 8,), -7, dtype=torch.int32, device="cuda")              # what lies before and behind is not looked at
    slots = around[off:off + n]
    slots.copy_(torch.arange(n))
    assert int(pkg.kv_append(rows, "mxfp4", planes, slots=slots)) == 0
    for i in sorted({0, 1, 2, 3, 4, n // 2, n - 5, n - 4, n - 3, n - 2, n - 1} & set(range(n))):
        for bad in (-1, n):
            slots[i] = bad
            assert int(pkg.kv_append(rows, "mxfp4", planes, slots=slots)) == 1
        slots[i] = i
    assert int(pkg.kv_append(rows, "mxfp4", planes, slots=slots)) == 0


@pytest.mark.parametrize("heads", [16, 32, 64])
@pytest.mark.parametrize("impl", ["tcgen05", "generic"])
def test_q_cast_with_values_beyond_the_given_maxima(pkg, impl, heads):
    """The caller's maxima may be those of another tensor: what lies beyond saturates, infinities included."""
    data = pkg.generate_input(3, 1, 200, seed=12, num_heads=heads, formats=("fp8",))
    q, kvd, _, ip, cfg = data
    parts, top = pkg.q_amax_parts(q).clone(), float(q.float().abs().max())
    wild, tame = q.clone(), q.clone()
    for (b, h, d), x in (((0, 3, 10), float("inf")), ((0, 9, 571), -3.0e38), ((1, 15, 511), float("-inf")), ((2, 0, 0), 1.0e30), ((2, 5, 64), 50 * top)):
        wild[b, h, d], tame[b, h, d] = x, top if x > 0 else -top
    run = lambda t: pkg.mla_decode(t, parts, "fp8", kvd["fp8"], ip, sm_scale=0.01, q_cast=True, impl=impl)
    assert torch.isfinite(run(wild).float()).all()
    assert torch.equal(run(wild), run(tame))
