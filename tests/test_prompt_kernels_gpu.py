"""Kernels that take many tokens of a prompt side by side, at the sizes where their tiles and chunks begin and end, against
the 64-bit run of ``fake_ops.FakeOps`` (the operations token by token) and against their own answers for the same rows in
other batches."""

from __future__ import annotations

import ctypes
import subprocess
import types

import pytest
import torch

from fake_ops import FakeOps
from mini_llm_runtime_b200 import ops
from mini_llm_runtime_b200.ops import AttentionBatch, cuda_ops

pytestmark = pytest.mark.gpu

DEVICE = "cuda:0"
FAKE = FakeOps()
UNIT = 2.0 ** -24          # relative rounding of one 32-bit operation


def cuda():
    return ops.current()


def generator(seed):
    return torch.Generator().manual_seed(seed)


def rnd(seed, *shape, std=1.0):
    return torch.randn(shape, generator=generator(seed)) * std


def spaced(tensor, extra=4):
    """The same rows as a column range of a wider product."""
    wide = torch.full((tensor.shape[0], tensor.shape[1] + 2 * extra), float("nan"))
    wide[:, extra:extra + tensor.shape[1]] = tensor
    return wide.to(DEVICE)[:, extra:extra + tensor.shape[1]]


def segments(lengths, slots, order=None):
    """A ragged batch; ``order`` lists the requests in the order of their rows (as listed by default)."""
    starts, at = [0] * len(lengths), 0
    for index in order or range(len(lengths)):
        starts[index] = at
        at += lengths[index]
    dev = lambda values: torch.tensor(values, dtype=torch.int32, device=DEVICE)      # noqa: E731
    return types.SimpleNamespace(
        seg_q_start=dev(starts), seg_q_len=dev(lengths), seg_slot=dev(slots), num_segments=len(lengths), max_q_len=max(lengths),
        segments=[types.SimpleNamespace(row_start=a, length=n, slot=s) for a, n, s in zip(starts, lengths, slots)])


def close(got, want, bound, what):
    """Relative error in the 2-norm, of the whole and of the worst row."""
    got, want = got.double().cpu().flatten(1), want.double().flatten(1)
    assert torch.isfinite(got).all(), what
    error = (got - want).norm(dim=1) / want.norm(dim=1).clamp_min(1e-3 * want.norm() / want.shape[0] ** 0.5)
    assert float(error.max()) <= bound, f"{what}: {float(error.max()):.2e}, allowed {bound:.2e}"


CHUNKED = [([1, 64, 65, 200], [3, 0, 2, 1], None), ([193, 128, 63, 1, 127], [4, 1, 0, 2, 3], [3, 1, 4, 0, 2]), ([321], [0], None)]


@pytest.mark.parametrize("mode", ["bonus", "forget"])
@pytest.mark.parametrize("heads,dim", [(3, 64), (2, 128)])
@pytest.mark.parametrize("lengths,slots,order", CHUNKED)
def test_gated_recurrences_in_chunks(mode, heads, dim, lengths, slots, order, monkeypatch):
    """Segments around the borders of chunks of 64 tokens, rows of requests in any order, decays of zero and one."""
    monkeypatch.setattr(cuda(), "GATED_ROWS", {64: (1, 1), 128: (1, 1)})      # short segments in chunks as well
    ctx, rows, n = segments(lengths, slots, order), sum(lengths), heads * dim
    r, k, v, gate = (rnd(i, rows, n, std=0.7) for i in range(4))
    raw, bias, weight = rnd(5, rows, n, std=0.5), rnd(6, n) * 2 - 2, 1 + rnd(7, n, std=0.1)
    raw[rows // 3, : n // 2], raw[rows // 2, n // 2:] = 60.0, -60.0        # decays of 0 and of 1 (lower bound and 1)
    aux = torch.rand(n, generator=generator(8)) if mode == "forget" else rnd(8, n, std=0.3)
    state = rnd(9, len(lengths), heads, dim, dim, std=0.5)
    want_state, got_state = state.double(), state.to(DEVICE)
    # a row's result is a sum over the channels of products that went through up to CHUNK decays; 64 roundings each way, and
    # the norm's and gate's own, stay below 200 roundings in the 2-norm of a row
    bound = 200 * UNIT
    for dtype in (torch.float32, torch.bfloat16):
        got_state.copy_(state)
        if mode == "bonus":
            want_state = state.double()
            want = FAKE.bonus_recurrence(*(t.double() for t in (r, k, v, raw, gate, bias, aux, weight)), 1e-6, want_state, ctx,
                                         heads, dim, torch.float32)
            got = cuda().bonus_recurrence(*(spaced(t) for t in (r, k, v, raw, gate)), *(t.to(DEVICE) for t in (bias, aux, weight)),
                                          1e-6, got_state, ctx, heads, dim, dtype)
        else:
            want_state = state.double()
            want = FAKE.forget_gate_recurrence(*(t.double() for t in (r, raw, v, bias, aux, weight[:dim])), 1e-6, want_state, ctx,
                                               heads, dim, dim, torch.float32)
            got = cuda().forget_gate_recurrence(*(spaced(t) for t in (r, raw, v)), bias.to(DEVICE), aux.to(DEVICE),
                                                weight[:dim].contiguous().to(DEVICE), 1e-6, got_state, ctx, heads, dim, dim, dtype)
        close(got, want, bound if dtype == torch.float32 else 2.0 ** -8, f"{mode} {dtype}")
        close(got_state.flatten(0, 1), want_state.flatten(0, 1), bound, f"{mode} state")


@pytest.mark.parametrize("n,k", [(130, 1023), (70, 2052), (33, 4101), (16400, 72)])
def test_products_of_the_32_bit_path_do_not_depend_on_the_rows_beside(n, k):
    """Row counts on both sides of every tile's edge; the sums' order is the same in every tile, so equal rows get equal bits."""
    x, w, bias = rnd(1, 1100, k), rnd(2, n, k, std=0.2), rnd(3, n)
    xd, wd, bd = x.to(DEVICE), w.to(DEVICE), bias.to(DEVICE)
    whole = cuda().linear(xd, wd, bd)
    # k products and sums, each rounded once: the error of an output is below k * UNIT times the sum of magnitudes
    magnitude = x.double().abs() @ w.double().abs().T + bias.double().abs()
    assert bool(((whole.double().cpu() - (x.double() @ w.double().T + bias.double())).abs() <= k * UNIT * magnitude).all())
    for rows in (1, 4, 16, 17, 32, 33, 63, 64, 65, 200):
        assert torch.equal(cuda().linear(xd[5:5 + rows].contiguous(), wd, bd), whole[5:5 + rows]), rows


@pytest.mark.parametrize("heads,n,groups", [(4, 64, 1), (6, 128, 2)])
@pytest.mark.parametrize("lengths,slots,order", CHUNKED)
def test_state_space_in_chunks(heads, n, groups, lengths, slots, order, monkeypatch):
    """Segments around the borders of chunks; decays from zero to one, among them tokens that neither keep nor forget."""
    monkeypatch.setattr(cuda(), "STATE_SPACE_CHUNK_ROWS", 1)      # short segments in chunks as well
    ctx, rows, inner = segments(lengths, slots, order), sum(lengths), heads * 64
    x, B, C, dt = rnd(1, rows, inner), rnd(2, rows, groups * n), rnd(3, rows, groups * n), rnd(4, rows, heads, std=2.0)
    dt[rows // 3], dt[rows // 2] = 90.0, -90.0
    dt_bias, a_log, skip = rnd(5, heads), rnd(6, heads), rnd(7, heads)
    state = rnd(8, len(lengths), heads, 64, n, std=0.5)
    want_state, got_state = state.double(), state.to(DEVICE)
    want = FAKE.state_space_scan(*(t.double() for t in (x, B, C, dt, dt_bias, a_log, skip)), want_state, ctx, heads, 64, n, groups)
    got = cuda().state_space_scan(*(spaced(t) for t in (x, B, C, dt)), *(t.to(DEVICE) for t in (dt_bias, a_log, skip)), got_state,
                                  ctx, heads, 64, n, groups)
    # sums of up to n + CHUNK products of numbers that went through up to CHUNK decays each
    close(got, want, 200 * UNIT, "state-space outputs")
    close(got_state.flatten(0, 1), want_state.flatten(0, 1), 200 * UNIT, "state-space state")


@pytest.mark.parametrize("heads,n,lengths", [(6, 64, [144, 65, 96, 143, 1, 16, 17]), (4, 128, [200, 70, 97, 64, 33, 2, 128]),      # halves
                                             (32, 128, [1000, 100, 66, 1]), (6, 64, [150, 64, 1, 33])])                          # whole
def test_state_space_of_short_portions_beside_chunks(heads, n, lengths):
    """Rows that go token by token beside the chunks' kernels, at once or in halves: the bits of a step of their own."""
    count, rows, inner = len(lengths), sum(lengths), heads * 64
    ctx = segments(lengths, list(reversed(range(count))), [*range(1, count), 0])
    x, B, C, dt = (spaced(t) for t in (rnd(1, rows, inner), rnd(2, rows, n), rnd(3, rows, n), rnd(4, rows, heads, std=2.0)))
    vectors, state = [rnd(i, heads).to(DEVICE) for i in (5, 6, 7)], rnd(8, count, heads, 64, n, std=0.5).to(DEVICE)
    whole = state.clone()
    y = cuda().state_space_scan(x, B, C, dt, *vectors, whole, ctx, heads, 64, n, 1)
    for part in ctx.segments:
        at, own = slice(part.row_start, part.row_start + part.length), state.clone()
        alone = cuda().state_space_scan(x[at], B[at], C[at], dt[at], *vectors, own, segments([part.length], [part.slot]), heads, 64, n, 1)
        assert torch.equal(alone, y[at]) and torch.equal(own[part.slot], whole[part.slot]), part.length


@pytest.mark.parametrize("heads,n,groups", [(2, 64, 1), (4, 128, 2)])
@pytest.mark.parametrize("where", ["x", "B", "C", "state", "before"])
@pytest.mark.parametrize("value", [float("inf"), float("nan"), 3.4e38])
def test_state_space_chunks_with_numbers_that_have_no_parts(heads, n, groups, where, value, monkeypatch):
    """One such number among ordinary ones goes by multiply-adds in its chunk: outputs that are no numbers where token by token has them, the
    others as there.  ``before``: a state that only later chunks see."""
    monkeypatch.setattr(cuda(), "STATE_SPACE_CHUNK_ROWS", 65)
    launched, load = [], cuda_ops.build.load_library
    monkeypatch.setattr(cuda_ops.build, "load_library", lambda name: launched.append(name) or load(name))
    lengths, slots = [130, 65], [1, 0]
    ctx, rows, inner = segments(lengths, slots), sum(lengths), heads * 64
    x, B, C, dt = rnd(1, rows, inner), rnd(2, rows, groups * n), rnd(3, rows, groups * n), rnd(4, rows, heads, std=0.5) - 3
    state = rnd(8, 2, heads, 64, n, std=0.5)
    {"x": x, "B": B, "C": C, "state": state[1, 0], "before": x}[where][70 if where in ("x", "B", "C") else 3, 5] = value
    vectors = rnd(5, heads), rnd(6, heads), rnd(7, heads)
    results = []
    for chunks in (False, True):
        cuda().use_state_space_chunks = chunks
        try:
            s = state.to(DEVICE)
            y = cuda().state_space_scan(*(spaced(t) for t in (x, B, C, dt)), *(v.to(DEVICE) for v in vectors), s, ctx, heads, 64, n, groups)
        finally:
            cuda().use_state_space_chunks = True
        results.append((y.cpu().double(), s.cpu().double()))
    assert [name for name in launched if name.startswith("state_space")] == ["state_space", "state_space_chunks"]
    for want, got in zip(*results):
        # beside 3.4e38 sums overflow in one order and not in the other; the outputs and states that it has no part in are ordinary
        if value != 3.4e38:
            assert torch.equal(torch.isfinite(got), torch.isfinite(want))
        normal = torch.isfinite(want) & (want.abs() < 1e30)
        assert float((got[normal] - want[normal]).norm()) <= 200 * UNIT * float(want[normal].norm())


def paged(lengths, before, visible, page_size, pools, seed):
    """Pools [pages, heads, page_size, entries] and the batch, on the CPU and on the device.  Page 0 belongs to nobody; it and every
    place that no row of its request sees (``visible(position, key)``) hold NaN, and pages without a visible key are given back."""
    need = [-(-(n + b) // page_size) for n, b in zip(lengths, before)]
    order = torch.randperm(sum(need), generator=generator(seed)) + 1
    table = torch.full((len(lengths), max(need)), -1, dtype=torch.int32)
    tensors = [torch.full((sum(need) + 1, heads, page_size, entries), float("nan"), dtype=torch.bfloat16) for heads, entries, _ in pools]
    at = 0
    for index, (n, b) in enumerate(zip(lengths, before)):
        for logical in range(need[index]):
            page = int(order[at])
            at += 1
            offsets = [o for o in range(page_size) if any(visible(p, logical * page_size + o) for p in range(b, b + n))]
            if offsets:
                table[index, logical] = page
                for k, (tensor, (heads, entries, std)) in enumerate(zip(tensors, pools)):
                    tensor[page, :, offsets] = rnd(seed + 100 * page + k, heads, len(offsets), entries, std=std).to(torch.bfloat16)
    starts = torch.tensor([sum(lengths[:i]) for i in range(len(lengths))], dtype=torch.int32)
    arrays, counts = cuda().plan_attention(lengths, before)
    cpu = dict(seg_q_start=starts, seg_q_len=torch.tensor(lengths, dtype=torch.int32), seg_pos0=torch.tensor(before, dtype=torch.int32),
               seg_slot=torch.arange(len(lengths), dtype=torch.int32), block_table=table)
    rest = dict(num_segments=len(lengths), max_q_len=max(lengths), max_kv_len=max(n + b for n, b in zip(lengths, before)), counts=counts)
    batch = AttentionBatch(**{k: v.to(DEVICE) for k, v in cpu.items()}, **rest,
                           plan={k: torch.from_numpy(v).to(DEVICE) for k, v in arrays.items()})
    return tensors, types.SimpleNamespace(**cpu, **rest), batch


# Probabilities, keys and values in bfloat16 (8 bits each), sums in 32: of the rounding errors only those of the probabilities and of
# the result are not the oracle's too, 2^-9 each at most and independent from key to key.
ATTENTION_BOUND = 2.0 ** -7


@pytest.mark.parametrize("dim,vdim,page_size", [(64, 128, 16), (128, 64, 8), (64, 64, 64), (128, 128, 32)])
@pytest.mark.parametrize("window,keep", [(70, 5), (0, 0), (129, 70)])
def test_differential_attention_of_prompts(dim, vdim, page_size, window, keep):
    """Portions around the 128 rows of an item, tiles of 64 keys around the kept positions and the window."""
    heads, kv_heads, lengths, before = 4, 2, [129, 5, 66, 4, 64], [0, 300, 100, 50, 64]
    seen = lambda p, j: j <= p and (not window or p - j < window or j < keep)      # noqa: E731
    pools, cpu, batch = paged(lengths, before, seen, page_size, [(kv_heads, 2 * dim, 1.0), (kv_heads, vdim, 0.7)], 3)
    q = rnd(5, sum(lengths), 2 * heads * dim).to(torch.bfloat16)
    args = (heads, kv_heads, dim, vdim, dim ** -0.5, window, keep, 0.4, 1e-6, 0.5)
    want = FAKE.differential_attention(q.float(), *(t.float() for t in pools), cpu, *args)
    got = cuda().differential_attention(q.to(DEVICE), *(t.to(DEVICE) for t in pools), batch, *args)
    torch.cuda.synchronize()
    cuda().raise_if_device_error()
    # the difference of two maps, brought to unit size: its share of their errors grows by what the difference lost
    close(got, want, 2 * ATTENTION_BOUND, "differential attention")


@pytest.mark.parametrize("heads,rank,rot,page_size", [(16, 512, 64, 16), (14, 256, 32, 16), (5, 384, 32, 64), (128, 64, 16, 8), (3, 48, 16, 32)])
@pytest.mark.parametrize("window", [0, 70])
@pytest.mark.parametrize("sinks", [False, True])
def test_latent_attention_of_prompts(heads, rank, rot, page_size, window, sinks):
    """Portions around the tokens of an item (128 / heads) and around tiles of 32 and 64 keys; latents in one piece and in halves."""
    lengths, before = [130, 2, 33, 9], [0, 300, 95, 31]
    seen = lambda p, j: j <= p and (not window or p - j < window)      # noqa: E731
    (pool,), cpu, batch = paged(lengths, before, seen, page_size, [(1, rank + rot, 1.0)], 7)
    q = rnd(6, sum(lengths), heads * (rank + rot), std=0.5).to(torch.bfloat16)
    sink = rnd(8, heads) if sinks else None
    args = (heads, rank, rot, 2.0 * (rank + rot) ** -0.5, window)
    want = FAKE.latent_attention(q.float(), pool.float(), cpu, *args, sink)
    got = cuda().latent_attention(q.to(DEVICE), pool.to(DEVICE), batch, *args, None if sink is None else sink.to(DEVICE))
    torch.cuda.synchronize()
    cuda().raise_if_device_error()
    close(got, want, ATTENTION_BOUND, "latent attention")


@pytest.mark.parametrize("heads,kv_heads,dim,vdim", [(16, 4, 128, 128), (14, 2, 64, 64), (3, 1, 64, 128), (6, 6, 128, 64)])
@pytest.mark.parametrize("mixed", [False, True])
def test_sigmoid_attention_of_prompts(heads, kv_heads, dim, vdim, mixed):
    """Head counts that fill no group of four, rows around the 16 of an entry, keys around tiles of 32 and a cut into chunks."""
    lengths, before = [33, 5, 17], [0, 402, 95]
    (k_pool, v_pool), cpu, batch = paged(lengths, before, lambda p, j: j <= p, 16, [(kv_heads, dim, 1.0), (kv_heads, vdim, 0.5)], 9)
    q = rnd(6, sum(lengths), heads * dim).to(torch.bfloat16)
    vectors = dict(distance=(torch.rand(heads, generator=generator(1)), torch.rand(heads, generator=generator(2))), score_bias=rnd(3, heads, std=0.3),
                   head_mix=torch.eye(heads) + rnd(4, heads, heads, std=0.1)) if mixed else {}
    args = (heads, kv_heads, dim, vdim, dim ** -0.5)
    want = FAKE.sigmoid_attention(q.float(), k_pool.float(), v_pool.float(), cpu, *args, **vectors)
    there = {k: tuple(t.to(DEVICE) for t in v) if isinstance(v, tuple) else v.to(DEVICE) for k, v in vectors.items()}
    got = cuda().sigmoid_attention(q.to(DEVICE), k_pool.to(DEVICE), v_pool.to(DEVICE), batch, *args, **there)
    close(got, want, ATTENTION_BOUND, "sigmoid attention")


def on_tcgen05(monkeypatch):
    """Every sigmoid attention of sizes that fit on tcgen05, whatever it costs; how many calls went there."""
    lib, calls = cuda_ops._declared_library("attention_sigmoid_tcgen05"), []
    kernel = lib.mlr_attention_sigmoid_tcgen05
    monkeypatch.setattr(cuda(), "_sigmoid_few", lambda *args: False, raising=False)
    monkeypatch.setattr(lib, "mlr_attention_sigmoid_tcgen05", lambda *args: calls.append(1) or kernel(*args))
    return calls


@pytest.mark.parametrize("heads,kv_heads,dim,vdim,page_size", [(16, 4, 128, 128, 8), (14, 2, 64, 64, 16), (9, 3, 128, 64, 64), (5, 1, 64, 128, 256),
                                                               (4, 4, 64, 64, 128)])
@pytest.mark.parametrize("lengths,before,limit", [
    ([129], [0], 0), ([16, 1, 8], [112, 640, 300], 0), ([1] * 7, [127, 128, 63, 64, 1000, 200, 500], 0), ([1] * 6, [2700, 3, 60, 127, 128, 11], 0),
    ([70, 260, 9, 1], [250, 0, 127, 383], 0), ([1, 30, 17], [64, 70, 111], 0), ([40, 3, 1], [210, 250, 192], 0),
    ([1] * 150 + [25], [40 + i % 88 for i in range(150)] + [100], 0), ([1] * 6, [20, 300, 64, 127, 0, 500], 1024)])
def test_sigmoid_attention_on_tcgen05(heads, kv_heads, dim, vdim, page_size, lengths, before, limit, monkeypatch):
    """Keys around tiles of 128 and their halves, rows around the 8 of half an entry, entries cut and whole, pages smaller and larger than a
    tile and its halves, heads that do not fill fours; steps of one and two tiles per entry, of more entries than CTAs, planned for a context limit as captured
    ones are; places that no row sees hold NaN.  Mixing factors large enough that what mixing in fewer
    than 32 bits would leave of the weights shows.  The second call finds the first one's scratch."""
    (k_pool, v_pool), cpu, batch = paged(lengths, before, lambda p, j: j <= p, page_size, [(kv_heads, dim, 1.0), (kv_heads, vdim, 0.5)], 11)
    batch.max_kv_len = max(limit, batch.max_kv_len)
    assert cuda().use_tcgen05_attention and cuda_ops.build.load_library("attention_sigmoid_tcgen05").mlr_attention_sigmoid_tcgen05_fits(
        heads, kv_heads, dim, vdim, page_size)
    q = rnd(6, sum(lengths), heads * dim).to(torch.bfloat16)
    vectors = dict(distance=(torch.rand(heads, generator=generator(1)), torch.rand(heads, generator=generator(2))), score_bias=rnd(3, heads, std=0.3),
                   head_mix=rnd(4, heads, heads))
    args = (heads, kv_heads, dim, vdim, dim ** -0.5)
    want = FAKE.sigmoid_attention(q.float(), k_pool.float(), v_pool.float(), cpu, *args, **vectors)
    there = {k: tuple(t.to(DEVICE) for t in v) if isinstance(v, tuple) else v.to(DEVICE) for k, v in vectors.items()}
    calls = on_tcgen05(monkeypatch)
    first = cuda().sigmoid_attention(q.to(DEVICE), k_pool.to(DEVICE), v_pool.to(DEVICE), batch, *args, **there)
    got = cuda().sigmoid_attention(q.to(DEVICE), k_pool.to(DEVICE), v_pool.to(DEVICE), batch, *args, **there)
    torch.cuda.synchronize()
    cuda().raise_if_device_error()
    assert len(calls) == 2
    # mixed weights and results are rounded to 8 bits, 2^-9 each at most; mixed with signs, weights lose size against the keys' sum of squares no
    # more than in ATTENTION_BOUND's own margin
    close(got, want, ATTENTION_BOUND, "sigmoid attention")
    assert torch.equal(first, got)


def test_a_kernel_compiled_to_other_registers_is_not_offered(tmp_path):
    """The shares of another launch than the compiler's: the sizes do not fit, so that calls go on to the kernel behind it."""
    source = (cuda_ops.build.CSRC / "attention_sigmoid_tcgen05.cu").read_text()
    shares = "SG_LAUNCH_REGISTERS = 168, SG_COMPUTE_REGISTERS = 208, SG_OTHER_REGISTERS = 88"
    assert shares in source
    (tmp_path / "other.cu").write_text(source.replace(shares, "SG_LAUNCH_REGISTERS = 160, SG_COMPUTE_REGISTERS = 200, SG_OTHER_REGISTERS = 80"))
    subprocess.run([cuda_ops.build.find_nvcc(), *cuda_ops.build.ARCH_FLAGS, *cuda_ops.build.COMMON_FLAGS, f"-I{cuda_ops.build.CSRC}", "-o",
                    str(tmp_path / "other.so"), str(tmp_path / "other.cu")], check=True)
    other, own = ctypes.CDLL(str(tmp_path / "other.so")), cuda_ops.build.load_library("attention_sigmoid_tcgen05")
    for dim, vdim in ((64, 64), (64, 128), (128, 64), (128, 128)):
        assert own.mlr_attention_sigmoid_tcgen05_fits(8, 2, dim, vdim, 16) == 1 and other.mlr_attention_sigmoid_tcgen05_fits(8, 2, dim, vdim, 16) == 0


def test_heads_mixed_by_parts_are_mixed_in_32_bits():
    """Weights that cancel in the mixing, to results that 16 bits of them would not show: twelve equal heads, factors whose sum is 2^-12."""
    heads, dim, rows = 12, 64, 40
    (k_pool, v_pool), cpu, batch = paged([rows], [100], lambda p, j: j <= p, 16, [(1, dim, 1.0), (1, dim, 0.5)], 12)
    q = rnd(6, rows, 1, dim).expand(rows, heads, dim).reshape(rows, heads * dim).to(torch.bfloat16)
    mix = rnd(4, heads, heads)
    mix[:, -1] += 2.0 ** -12 - mix.double().sum(1).float()
    mix[:, -1] += (2.0 ** -12 - mix.double().sum(1)).float()
    args = (heads, 1, dim, dim, dim ** -0.5)
    sums = mix.double().sum(1)
    plain = FAKE.sigmoid_attention(q.double(), k_pool.double(), v_pool.double(), cpu, *args).double().view(rows, heads, dim)
    want = (plain[:, :1] * sums[None, :, None]).reshape(rows, heads * dim)
    got = cuda().sigmoid_attention(q.to(DEVICE), k_pool.to(DEVICE), v_pool.to(DEVICE), batch, *args, head_mix=mix.to(DEVICE))
    # a mixed weight is a sum of twelve products of numbers around one, each rounded to 2^-24 (the tensor cores' sums drop as much), beside a result
    # of 2^-12 / 2: below 12 * 2 * 2^-24 / 2^-13 = 2^-6.4 of it, independent from key to key
    close(got, want, ATTENTION_BOUND + 2.0 ** -6.4, "mixed weights")


@pytest.mark.parametrize("heads,dim", [(12, 64), (16, 128)])
def test_heads_mixed_by_parts_lose_no_more_than_multiply_adds(heads, dim, monkeypatch):
    """Equal heads, factors whose sum is 2^-17: what the mixing lost of 32 bits shows in the 8 bits of the mixed weights."""
    rows = 300
    (k_pool, v_pool), cpu, batch = paged([rows], [0], lambda p, j: j <= p, 16, [(1, dim, 1.0), (1, dim, 0.5)], 12)
    q = rnd(6, rows, 1, dim).expand(rows, heads, dim).reshape(rows, heads * dim).to(torch.bfloat16)
    mix = rnd(4, heads, heads)
    for _ in range(3):
        mix[:, -1] += (2.0 ** -17 - mix.double().sum(1)).float()
    args = (heads, 1, dim, dim, dim ** -0.5)
    plain = FAKE.sigmoid_attention(q.double(), k_pool.double(), v_pool.double(), cpu, *args).double().view(rows, heads, dim)
    want = (plain[:, :1] * mix.double().sum(1)[None, :, None]).reshape(rows, heads * dim)
    calls, errors = on_tcgen05(monkeypatch), []
    for wide in (False, True):
        monkeypatch.setattr(cuda(), "use_tcgen05_attention", wide)
        got = cuda().sigmoid_attention(q.to(DEVICE), k_pool.to(DEVICE), v_pool.to(DEVICE), batch, *args, head_mix=mix.to(DEVICE))
        errors.append(float((got.double().cpu() - want).norm() / want.norm()))
    assert len(calls) == 1
    # a chain of multiply-adds rounds once per head; products of whole parts are cut once, by half a place on average
    assert 2.0 ** -8 < errors[0] and errors[1] <= 0.5 * errors[0], errors


@pytest.mark.parametrize("heads,kv_heads,dim", [(16, 4, 128), (14, 2, 64)])
def test_sigmoid_attention_of_long_contexts(heads, kv_heads, dim, monkeypatch):
    """Thousands of keys summed in one accumulator: as near to 64 bits as sums of up to 384 keys that are added in 32 bits."""
    rows, before, take = 2048, 6000, 128
    (k_pool, v_pool), cpu, batch = paged([rows], [before], lambda p, j: j <= p, 16, [(kv_heads, dim, 1.0), (kv_heads, dim, 0.6)], 13)
    q = rnd(6, rows, heads * dim).to(torch.bfloat16).to(DEVICE)
    bias, mix = rnd(3, heads, std=0.3).to(DEVICE), (torch.eye(heads) + rnd(4, heads, heads, std=0.1)).to(DEVICE)
    j = torch.arange(rows + before, device=DEVICE)
    keys, values = (pool.to(DEVICE)[cpu.block_table[0].to(DEVICE).long()[j // 16], :, j % 16].double().repeat_interleave(heads // kv_heads, 1)
                    for pool in (k_pool, v_pool))
    scores = torch.einsum("rhd,nhd->rhn", q[-take:].view(take, heads, dim).double(), keys) * dim ** -0.5 + bias.double()[:, None]
    seen = (j[None] <= before + rows - take + torch.arange(take, device=DEVICE)[:, None])[:, None]
    want = torch.einsum("rhn,nhd->rhd", torch.einsum("hg,rgn->rhn", mix.double(), torch.sigmoid(scores) * seen), values).flatten(1)
    calls, errors = on_tcgen05(monkeypatch), []
    for wide in (False, True):
        monkeypatch.setattr(cuda(), "use_tcgen05_attention", wide)
        got = cuda().sigmoid_attention(q, k_pool.to(DEVICE), v_pool.to(DEVICE), batch, heads, kv_heads, dim, dim, dim ** -0.5, score_bias=bias, head_mix=mix)
        errors.append(float((got[-take:].double() - want).norm() / want.norm()))
    assert len(calls) == 1
    # both are the roundings of weights and results to 8 bits, some 2^-8.8; of 200,000 numbers their means of squares differ by a few in a thousand
    assert errors[1] <= 1.005 * errors[0], errors


@pytest.mark.parametrize("heads,dim,vdim", [(2, 128, 128), (3, 64, 72)])
@pytest.mark.parametrize("lengths,slots,order", [([1, 512, 513, 1100], [3, 0, 2, 1], None), ([515, 3, 1030], [1, 2, 0], [2, 0, 1])])
def test_matrix_memory_of_long_portions(heads, dim, vdim, lengths, slots, order):
    """Segments of many chunks side by side, rows of requests in any order, gates that forget and keep everything: as with one chunk behind the
    other (which the 64-bit oracle vouches for elsewhere), whose products are the same and whose sums another order."""
    ctx, rows = segments(lengths, slots, order), sum(lengths)
    assert cuda()._memory_chunks_fit(dim, vdim) and beside(ctx, rows, vdim)
    q, k, v, gate = rnd(1, rows, heads * dim), rnd(2, rows, heads * dim), rnd(3, rows, heads * vdim), rnd(4, rows, heads * vdim)
    i_raw, f_raw = rnd(5, rows, heads), rnd(6, rows, heads, std=2.0)
    f_raw[rows // 3], f_raw[rows // 2] = -80.0, 80.0
    bias, weight = torch.zeros(heads), 1 + rnd(7, heads * vdim, std=0.1)
    state, maximum = rnd(8, len(lengths), heads, vdim + 1, dim, std=0.5), rnd(9, len(lengths), heads)
    results = []
    for together in (False, True):
        cuda().use_memory_side_by_side = together
        try:
            s, m = state.to(DEVICE), maximum.to(DEVICE)
            out = cuda().matrix_memory(*(spaced(t, 8) for t in (q, k, v, i_raw, f_raw)), bias.to(DEVICE), bias.to(DEVICE) + 3, 15.0, 1e-6,
                                       spaced(gate, 8), weight.to(DEVICE), 1e-6, s, m, ctx, heads, dim, vdim, torch.bfloat16)
        finally:
            cuda().use_memory_side_by_side = True
        results.append((out.cpu(), s.cpu(), m.cpu()))
    (out, s, m), (want, want_s, want_m) = results[1], results[0]
    assert torch.equal(m, want_m)
    close(s.flatten(0, 1), want_s.flatten(0, 1), 200 * UNIT, "state")      # sums of 64 products at a time, once per chunk
    close(out, want, 2.0 ** -8, "output")


def gated(mode, dtype, inputs, weight, aux, bias, state, ctx, heads, dim):
    """One call of a gated recurrence on the rows ``inputs`` (r, k, v, gate, raw); the state is advanced in place."""
    r, k, v, gate, raw = inputs
    if mode == "bonus":
        return cuda().bonus_recurrence(r, k, v, raw, gate, bias, aux, weight, 1e-6, state, ctx, heads, dim, dtype)
    return cuda().forget_gate_recurrence(r, raw, v, bias, aux, weight[:dim].contiguous(), 1e-6, state, ctx, heads, dim, dim, dtype)


# requests whose portions are too short for chunks, each list beside a portion that is long enough
SHORT = [[1, 1, 1], [3, 1, 31], [32, 1, 63], [1, 100, 127], [1, 159, 191]]


@pytest.mark.parametrize("mode", ["bonus", "forget"])
@pytest.mark.parametrize("heads,dim", [(3, 64), (2, 128)])
@pytest.mark.parametrize("short", SHORT)
@pytest.mark.parametrize("beside", [192, 400])
def test_a_short_portion_of_a_gated_recurrence_is_the_same_beside_a_long_one(mode, heads, dim, short, beside):
    n, rows = heads * dim, sum(short)
    inputs = [rnd(i, rows + beside, n, std=0.7).to(DEVICE) for i in range(5)]
    bias, weight, aux = (t.to(DEVICE) for t in (rnd(6, n) * 2 - 2, 1 + rnd(7, n, std=0.1), torch.rand(n, generator=generator(8))))
    state = rnd(9, len(short) + 1, heads, dim, dim, std=0.5).to(DEVICE)
    results = []
    for lengths in (short, short + [beside]):
        s = state.clone()
        out = gated(mode, torch.float32, [t[:sum(lengths)].contiguous() for t in inputs], weight, aux, bias, s,
                    segments(lengths, list(range(len(lengths)))), heads, dim)
        results.append((out[:rows], s[:len(short)]))
    assert torch.equal(results[0][0], results[1][0]) and torch.equal(results[0][1], results[1][1])


@pytest.mark.parametrize("heads,n,groups", [(4, 64, 1), (6, 128, 2)])
@pytest.mark.parametrize("short", SHORT)
@pytest.mark.parametrize("beside", [192, 400])
def test_a_short_portion_of_the_state_space_recurrence_is_the_same_beside_a_long_one(heads, n, groups, short, beside):
    rows = sum(short)
    full = [rnd(i, rows + beside, width).to(DEVICE) for i, width in enumerate((heads * 64, groups * n, groups * n, heads))]
    vectors = [rnd(i, heads).to(DEVICE) for i in (5, 6, 7)]
    state = rnd(8, len(short) + 1, heads, 64, n, std=0.5).to(DEVICE)
    results = []
    for lengths in (short, short + [beside]):
        s = state.clone()
        out = cuda().state_space_scan(*(t[:sum(lengths)].contiguous() for t in full), *vectors, s,
                                      segments(lengths, list(range(len(lengths)))), heads, 64, n, groups)
        results.append((out[:rows], s[:len(short)]))
    assert torch.equal(results[0][0], results[1][0]) and torch.equal(results[0][1], results[1][1])


def test_recurrences_take_batches_without_lengths_on_the_host():
    """A context that only says how many requests there are and which is the longest."""
    lengths, heads, n = [400, 1, 100, 193], 4, 64
    ctx = segments(lengths, [1, 0, 3, 2])
    bare = types.SimpleNamespace(**{k: v for k, v in vars(ctx).items() if k != "segments"})
    x, B, C, dt = (rnd(i, sum(lengths), width).to(DEVICE) for i, width in enumerate((heads * 64, n, n, heads)))
    vectors = [rnd(i, heads).to(DEVICE) for i in (5, 6, 7)]
    inputs = [rnd(i, sum(lengths), heads * 64, std=0.7).to(DEVICE) for i in range(5)]
    weight, aux, bias = (rnd(i, heads * 64).to(DEVICE) for i in (10, 11, 12))
    results = []
    for context in (ctx, bare):
        s = rnd(8, 4, heads, 64, n, std=0.5).to(DEVICE)
        y = cuda().state_space_scan(x, B, C, dt, *vectors, s, context, heads, 64, n, 1)
        g = rnd(9, 4, heads, 64, 64, std=0.5).to(DEVICE)
        out = gated("bonus", torch.bfloat16, inputs, weight, aux, bias, g, context, heads, 64)
        results.append((y, s, out, g))
    assert all(torch.equal(a, b) for a, b in zip(*results))


@pytest.mark.parametrize("heads,n", [(4, 64), (2, 128)])
@pytest.mark.parametrize("value", [float("inf"), float("nan")])
@pytest.mark.parametrize("at", [70, 127, 199])
def test_a_token_that_is_no_number_leaves_the_tokens_before_it_alone(heads, n, value, at):
    lengths = [200, 193]
    x, B, C, dt = (rnd(i, sum(lengths), width) for i, width in enumerate((heads * 64, n, n, heads)))
    vectors = [rnd(i, heads).to(DEVICE) for i in (5, 6, 7)]
    results = []
    for poisoned in (False, True):
        if poisoned:
            x[at], B[at], C[at], dt[at] = value, value, value, value
        s = torch.zeros(2, heads, 64, n, device=DEVICE)
        y = cuda().state_space_scan(*(t.to(DEVICE) for t in (x, B, C, dt)), *vectors, s, segments(lengths, [0, 1]), heads, 64, n, 1)
        results.append((y, s))
    (want, want_s), (got, got_s) = results
    assert torch.equal(got[:at], want[:at]) and torch.equal(got[200:], want[200:]) and torch.equal(got_s[1], want_s[1])
    assert not torch.isfinite(got[at]).any()


def relative(got, want):
    return float((got.double().cpu() - want.double()).norm() / want.double().norm())


@pytest.mark.parametrize("heads,rank,rot", [(16, 512, 64), (14, 256, 32)])
def test_latent_prompts_are_as_close_to_64_bits_on_either_kernel(heads, rank, rot):
    """The probabilities' rounding to 16 bits is all of the error, and the same error in both kernels; the 2-norm over 3e5 and more outputs
    varies by far less than the two percent left to it."""
    lengths, before = [150, 90], [200, 0]
    (pool,), cpu, batch = paged(lengths, before, lambda p, j: j <= p, 16, [(1, rank + rot, 1.0)], 7)
    q = rnd(6, sum(lengths), heads * (rank + rot), std=0.5).to(torch.bfloat16)
    args = (heads, rank, rot, 0.08, 0)
    want = FAKE.latent_attention(q.float(), pool.float(), cpu, *args, None)
    errors = []
    for tcgen05 in (False, True):
        cuda().use_tcgen05_attention = tcgen05
        try:
            errors.append(relative(cuda().latent_attention(q.to(DEVICE), pool.to(DEVICE), batch, *args, None), want))
        finally:
            cuda().use_tcgen05_attention = True
    print("error mma.sync, tcgen05:", errors)
    assert errors[1] <= 1.02 * errors[0], errors


@pytest.mark.parametrize("dim,vdim", [(64, 128), (128, 128)])
@pytest.mark.parametrize("window", [0, 120])
def test_differential_prompts_are_as_close_to_64_bits_on_either_kernel(dim, vdim, window):
    """As above; the outputs' own rounding to 16 bits is in both errors."""
    heads, kv_heads, lengths, before, keep = 6, 2, [200, 90], [150, 0], 4
    seen = lambda p, j: j <= p and (not window or p - j < window or j < keep)      # noqa: E731
    pools, cpu, batch = paged(lengths, before, seen, 16, [(kv_heads, 2 * dim, 1.0), (kv_heads, vdim, 0.7)], 3)
    q = rnd(5, sum(lengths), 2 * heads * dim).to(torch.bfloat16)
    args = (heads, kv_heads, dim, vdim, dim ** -0.5, window, keep, 0.4, 1e-6, 0.5)
    want = FAKE.differential_attention(q.float(), *(t.float() for t in pools), cpu, *args)
    errors = []
    for tcgen05 in (False, True):
        cuda().use_tcgen05_attention = tcgen05
        try:
            errors.append(relative(cuda().differential_attention(q.to(DEVICE), *(t.to(DEVICE) for t in pools), batch, *args), want))
        finally:
            cuda().use_tcgen05_attention = True
    print("error mma.sync, tcgen05:", errors)
    assert errors[1] <= 1.02 * errors[0], errors


@pytest.mark.parametrize("heads,kv_heads,dim,vdim", [(9, 9, 128, 128), (11, 11, 128, 64), (8, 8, 64, 64), (15, 3, 64, 64), (13, 1, 128, 128)])
def test_sigmoid_attention_of_many_key_heads(heads, kv_heads, dim, vdim):
    """Sizes whose tiles come close to an SM's shared memory, all on the tensor cores."""
    from mini_llm_runtime_b200.ops import build
    assert build.load_library("attention_sigmoid_mma").mlr_attention_sigmoid_mma_fits(heads, kv_heads, dim, vdim) == 1
    test_sigmoid_attention_of_prompts(heads, kv_heads, dim, vdim, True)
    test_sigmoid_attention_of_prompts(heads, kv_heads, dim, vdim, False)


def test_long_sums_of_many_rows_keep_their_scratch_bounded():
    """4,000 rows in four parts of every sum: the rows in blocks whose parts fit the bound, with the bits of a call of their own."""
    m, n, k = 4000, 3000, 4100
    x, w, bias = (t.to(DEVICE) for t in (rnd(1, m, k), rnd(2, n, k, std=0.2), rnd(3, n)))
    torch.cuda.synchronize()
    torch.cuda.reset_peak_memory_stats()
    start = torch.cuda.memory_allocated()
    whole = cuda().linear(x, w, bias)
    extra = torch.cuda.max_memory_allocated() - start - whole.numel() * 4
    assert extra <= 129 << 20, extra
    for first, rows in ((0, 64), (1300, 500), (3937, 63)):
        assert torch.equal(cuda().linear(x[first:first + rows].contiguous(), w, bias), whole[first:first + rows]), first


@pytest.mark.parametrize("width,inner", [(72, 64), (200, 192), (512, 128)])
@pytest.mark.parametrize("activation", ["silu", "gelu_tanh"])
@pytest.mark.parametrize("weigh_input", [False, True])
@pytest.mark.parametrize("others", [0, 300])
def test_experts_of_any_number_of_rows(width, inner, activation, weigh_input, others):
    """Rows of an expert around the multiples of 16 and 32 of an MMA and a copy, of the 64 and 128 of half a tile and a tile, none at all; columns
    that fill no copy of 64, weight rows that fill no tile of 256, so many tiles that a CTA takes several, and so few that the down product's are half as high."""
    counts = [1, 15, 0, 16, 17, 31, 33, 63, 64, 65, 96, 127, 128, 129, 255, 256, 257] + [3] * others
    experts, rows = len(counts), sum(counts)
    chosen = torch.repeat_interleave(torch.arange(experts), torch.tensor(counts))[torch.randperm(rows, generator=generator(1))]
    x, weights = rnd(2, rows, width).to(torch.bfloat16), torch.rand(rows, 1, generator=generator(3)) + 0.5
    gate_up, down = (rnd(4, experts, 2 * inner, width, std=width ** -0.5).to(torch.bfloat16),
                     rnd(5, experts, width, inner, std=inner ** -0.5).to(torch.bfloat16))
    got = cuda().routed_experts(x.to(DEVICE), chosen[:, None].int().to(DEVICE), weights.to(DEVICE), gate_up.to(DEVICE), down.to(DEVICE), 64,
                                activation, weigh_input)
    torch.cuda.synchronize()
    cuda().raise_if_device_error()
    act = torch.nn.functional.silu if activation == "silu" else lambda z: torch.nn.functional.gelu(z, approximate="tanh")
    want = torch.zeros(rows, width, dtype=torch.float64)
    for e in range(experts):
        mine = chosen == e
        both = (x[mine].double() @ gate_up[e].double().T * (weights[mine].double() if weigh_input else 1.0)).view(-1, inner // 64, 2, 64)
        want[mine] = (act(both[:, :, 0]) * both[:, :, 1]).flatten(1) @ down[e].double().T * (1.0 if weigh_input else weights[mine].double())
    # the hidden numbers' rounding to 8 bits, 2^-9 each at most and independent
    close(got, want, 2.0 ** -8, "experts")


@pytest.mark.parametrize("rows,top,experts", [(2048, 6, 64), (1500, 7, 33), (1366, 6, 128), (9000, 1, 40)])
def test_pairs_sorted_by_expert_in_several_turns(rows, top, experts):
    """More than the 8,192 choices that the sort's threads hold at once, more experts than a warp has lanes; one expert gets none.  Weights of
    few bits and expert matrices that only scale, so that every output is exact in 32 bits."""
    width = 128
    x = torch.randint(-8, 9, (rows, width), generator=generator(1)).to(torch.bfloat16)
    chosen = torch.stack([torch.randperm(experts - 1, generator=generator(10 + r))[:top] for r in range(rows)]).int()
    weights = torch.randint(1, 5, (rows, top), generator=generator(2)).float() / 4
    # gate rows of zeros but for a constant would need a bias; silu(g) * u with g = x and u = x is the same for every expert, and down
    # scales it by a power of two of the expert's own
    eye = torch.eye(width)
    gate_up = torch.cat([torch.cat([eye[i:i + 64], eye[i:i + 64]]) for i in range(0, width, 64)])[None].expand(experts, -1, -1)
    scale = 2.0 ** (torch.arange(experts) % 8 - 4).float()
    down = eye[None] * scale[:, None, None]
    got = cuda().routed_experts(x.to(DEVICE), chosen.to(DEVICE), weights.to(DEVICE), gate_up.to(torch.bfloat16).contiguous().to(DEVICE),
                                down.to(torch.bfloat16).contiguous().to(DEVICE), 64)
    f = x.double()
    hidden = f * torch.sigmoid(f) * f
    want = hidden * (weights.double() * scale.double()[chosen.long()]).sum(1, keepdim=True)
    # hidden is rounded to 16 bits once, with the approximate exponential before
    assert bool(((got.double().cpu() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-6).all())


@pytest.mark.parametrize("lengths,slots,order", [([1, 512, 1100], [2, 0, 1], None), ([1030, 3], [1, 0], [1, 0])])
def test_matrix_memory_of_long_portions_against_64_bits(lengths, slots, order):
    heads, dim, vdim = 2, 64, 64
    ctx, rows = segments(lengths, slots, order), sum(lengths)
    assert beside(ctx, rows, vdim)
    q, k, v, gate = (rnd(i, rows, heads * 64) for i in range(4))
    i_raw, f_raw = rnd(5, rows, heads), rnd(6, rows, heads, std=2.0)
    f_raw[rows // 3], f_raw[rows // 2] = -80.0, 80.0
    bias, weight = torch.zeros(heads), 1 + rnd(7, heads * vdim, std=0.1)
    state, maximum = rnd(8, len(lengths), heads, vdim + 1, dim, std=0.5), rnd(9, len(lengths), heads)
    # the kernel's products take q, k and v rounded to bfloat16
    q, k, v = (t.to(torch.bfloat16).float() for t in (q, k, v))
    s64, m64 = state.double(), maximum.double()
    want = FAKE.matrix_memory(*(t.double() for t in (q, k, v, i_raw, f_raw, bias, bias + 3)), 15.0, 1e-6, gate.double(), weight.double(), 1e-6,
                              s64, m64, ctx, heads, dim, vdim, torch.float64)
    s, m = state.to(DEVICE), maximum.to(DEVICE)
    got = cuda().matrix_memory(*(spaced(t, 8) for t in (q, k, v, i_raw, f_raw)), bias.to(DEVICE), bias.to(DEVICE) + 3, 15.0, 1e-6,
                               spaced(gate, 8), weight.to(DEVICE), 1e-6, s, m, ctx, heads, dim, vdim, torch.bfloat16)
    # 32-bit sums over up to 18 chunks, whose decays and products are rounded 64 times each at most; the output in 16 bits
    close(s.flatten(0, 1), s64.flatten(0, 1), 2000 * UNIT, "state")
    close(got, want, 2.0 ** -8, "output")


@pytest.mark.parametrize("heads,dim,vdim", [(1, 64, 8), (3, 128, 88), (2, 64, 96), (2, 128, 128)])
@pytest.mark.parametrize("lengths,slots,order", [([129, 1, 64, 65], [0, 3, 2, 1], None), ([63, 192, 128, 2], [1, 0, 3, 2], [2, 1, 3, 0])])
def test_matrix_memory_side_by_side(heads, dim, vdim, lengths, slots, order):
    """Portions of one chunk, one row more, one less and several beside each other, few and many value channels: as one chunk behind the other.  A number
    that is none leaves the rows before it as they are."""
    ctx, rows = segments(lengths, slots, order), sum(lengths)
    assert beside(ctx, rows, vdim)
    q, k, v, gate = rnd(1, rows, heads * dim), rnd(2, rows, heads * dim), rnd(3, rows, heads * vdim), rnd(4, rows, heads * vdim)
    i_raw, f_raw = rnd(5, rows, heads), rnd(6, rows, heads, std=2.0)
    gate[5], gate[6], gate[7] = -200.0, 200.0, -87.0
    bias, weight = torch.zeros(heads), 1 + rnd(7, heads * vdim, std=0.1)
    state, maximum = rnd(8, len(lengths), heads, vdim + 1, dim, std=0.5), rnd(9, len(lengths), heads)

    def call(together, v):
        cuda().use_memory_side_by_side = together
        try:
            s, m = state.to(DEVICE), maximum.to(DEVICE)
            out = cuda().matrix_memory(*(spaced(t, 8) for t in (q, k, v, i_raw, f_raw)), bias.to(DEVICE), bias.to(DEVICE) + 3, 15.0, 1e-6,
                                       spaced(gate, 8), weight.to(DEVICE), 1e-6, s, m, ctx, heads, dim, vdim, torch.bfloat16)
        finally:
            cuda().use_memory_side_by_side = True
        return out.cpu(), s.cpu(), m.cpu()

    (out, s, m), (want, want_s, want_m) = call(True, v), call(False, v)
    assert torch.equal(m, want_m)
    close(s.flatten(0, 1), want_s.flatten(0, 1), 200 * UNIT, "state")      # sums of 64 products at a time, once per chunk
    close(out, want, 2.0 ** -8, "output")
    last = int(ctx.seg_q_start[lengths.index(max(lengths))]) + max(lengths) - 1      # of the longest portion, in a block of 16 rows of its own
    broken = v.clone()
    broken[last] = float("nan")
    after = call(True, broken)[0]
    kept = torch.arange(rows) != last
    kept[last - (max(lengths) - 1) % 16:last] = False      # rows of the same block meet it with a weight of nothing
    assert torch.equal(after[kept], out[kept]) and bool(after[last].isnan().any())


@pytest.mark.parametrize("heads,dim,vdim", [(64, 128, 128), (64, 64, 96)])
@pytest.mark.parametrize("what", ["state", "state and tokens"])
def test_matrix_memory_side_by_side_loses_no_bits_of_its_sums(heads, dim, vdim, what):
    """Sums that cancel to some 2^-18 of their products, which shows in 16 bits what was lost of 32: no more than one chunk behind the other loses.
    A head's norm takes the small sums to ordinary size."""
    rows, ctx = 192, segments([192], [0])
    query, k, v = (rnd(i, *shape).to(torch.bfloat16).double() for i, shape in ((1, (heads, dim)), (2, (rows, heads, dim)), (3, (rows, heads, vdim))))
    along = query / (query * query).sum(1, keepdim=True)
    state = rnd(4, heads, vdim + 1, dim).double()
    state -= torch.einsum("hcd,hd->hc", state, query)[..., None] * along[:, None]      # across the query
    rest = rnd(5, heads, vdim + 1) * dim ** 0.5 * 2.0 ** -18
    i_raw, maximum, take = torch.full((rows, heads), -15.0), torch.full((1, heads), 15.0), slice(0, 64)      # tokens write e^-30
    if what == "state":
        v.zero_()
    else:                                       # the state takes back what a chunk's tokens write, as its last row reads them
        i_raw, maximum, take = torch.zeros(rows, heads), torch.zeros(1, heads), slice(63, 64)
        written = torch.einsum("shd,hd,shc->hc", k[:64], query, torch.cat([v[:64], torch.ones(64, heads, 1)], 2))
        rest = rest * 8 - written
    state = (state + rest[..., None] * along[:, None]).float()[None]
    q, k, v = query.flatten().expand(rows, -1).float().contiguous(), k.flatten(1).float(), v.flatten(1).float()
    gate, weight = torch.zeros(rows, heads * vdim), torch.ones(heads * vdim)
    f_raw, zero = torch.full((rows, heads), 200.0), torch.zeros(heads)      # kept whole
    s64 = state.double()
    want = FAKE.matrix_memory(*(t.double() for t in (q, k, v, i_raw, f_raw, zero, zero)), 100.0, 1e-6, gate.double(), weight.double(), 1e-30,
                              s64, maximum.double(), types.SimpleNamespace(**{**vars(ctx), "seg_slot": ctx.seg_slot.cpu()}), heads, dim, vdim, torch.float64)
    errors, take = [], slice(0, 64) if what == "state" else slice(63, 64)
    for together in (False, True):
        cuda().use_memory_side_by_side = together
        try:
            got = cuda().matrix_memory(*(t.to(DEVICE) for t in (q, k, v, i_raw, f_raw, zero, zero)), 100.0, 1e-6, gate.to(DEVICE), weight.to(DEVICE),
                                       1e-30, state.to(DEVICE), maximum.to(DEVICE), ctx, heads, dim, vdim, torch.bfloat16)
        finally:
            cuda().use_memory_side_by_side = True
        errors.append(float((got.double().cpu() - want)[take].norm() / want[take].norm()))
    # 2^-18 of a sum's 24 bits leave six.  Thousands of numbers that were lost alike: the two means of squares differ by a few in a hundred by chance
    assert 2.0 ** -8 < errors[0] and errors[1] <= 1.03 * errors[0], errors


@pytest.mark.parametrize("heads,dim,vdim", [(3, 128, 128), (2, 64, 72)])
def test_matrix_memory_of_decoded_rows_beside_a_portion(heads, dim, vdim):
    """Decoded rows have the bits of a step of their own with q, k and v in 16 bits, and cost no chunk's scratch; a portion's bits are those of a step of its
    own."""
    lengths = [1, 1, 130] + [1] * 61 + [2, 200, 1]
    count = len(lengths)
    order = torch.randperm(count, generator=generator(1)).tolist()
    ctx, rows = segments(lengths, torch.randperm(count, generator=generator(2)).tolist(), order), sum(lengths)
    q, k, v, gate = rnd(1, rows, heads * dim), rnd(2, rows, heads * dim), rnd(3, rows, heads * vdim), rnd(4, rows, heads * vdim)
    i_raw, f_raw = rnd(5, rows, heads), rnd(6, rows, heads, std=2.0)
    inputs = [spaced(t, 8) for t in (q, k, v, i_raw, f_raw, gate)]
    half = [spaced(t.to(torch.bfloat16).float(), 8) for t in (q, k, v)] + inputs[3:]
    bias, weight = torch.zeros(heads, device=DEVICE), (1 + rnd(7, heads * vdim, std=0.1)).to(DEVICE)
    state, maximum = rnd(8, count, heads, vdim + 1, dim, std=0.5).to(DEVICE), rnd(9, count, heads).to(DEVICE)

    def call(take, ctx, inputs):
        s, m = state.clone(), maximum.clone()
        rows = [t[take] for t in inputs]
        torch.cuda.synchronize()
        torch.cuda.reset_peak_memory_stats()
        start = torch.cuda.memory_allocated()
        out = cuda().matrix_memory(*rows[:5], bias, bias + 3, 15.0, 1e-6, rows[5], weight, 1e-6, s, m, ctx, heads, dim, vdim, torch.bfloat16)
        return out, s, m, torch.cuda.max_memory_allocated() - start

    out, s, m, extra = call(slice(None), ctx, inputs)
    chunks = 3 + 1 + 4
    assert extra <= chunks * heads * ((vdim + 1) * dim + 1) * 4 + rows * heads * (16 + 2 * vdim) + 4096, extra
    for part in ctx.segments:
        at = slice(part.row_start, part.row_start + part.length)
        own = call(at, segments([part.length], [part.slot]), half)
        if part.length != 2:                    # two rows alone go token by token
            assert torch.equal(own[0], out[at]) and torch.equal(own[1][part.slot], s[part.slot]), part.length
        assert torch.equal(own[2][part.slot], m[part.slot]), part.length


def beside(ctx, rows, vdim):
    from mini_llm_runtime_b200.ops import build
    return build.load_library("matrix_memory").mlr_matrix_memory_side_by_side(cuda()._chunks_from(ctx, rows, 1), ctx.num_segments, int(ctx.max_q_len), vdim)


# Tiles of 128 outputs, of 16, 32, 64 and 128 rows, blocks of 64 k; 1, 2, 4 and 8 parts of the sums over k; more tiles than SMs, few rows too.
@pytest.mark.parametrize("n,k", [(1024, 832), (1152, 896), (896, 4864), (130, 6148), (7000, 132), (9728, 200), (33, 30000), (20100, 132)])
@pytest.mark.parametrize("m", [1, 16, 17, 32, 33, 64, 65, 300])
def test_products_in_parts(m, n, k):
    """32-bit products on the tensor cores: dropped products of parts are below 2^-26 of sum |x||w|, a block's accumulator drops up to
    2^-23 of its sum at some dozen steps, each block and part is one 32-bit addition; rows keep their bits in other batches."""
    x, w, bias = (t.to(DEVICE) for t in (rnd(m, m, k), rnd(2, n, k, std=0.2), rnd(3, n)))
    ops_ = cuda()
    assert ops_._split_fits(x, w) == (n * k >= ops_.SPLIT_WEIGHT)
    got, shifted = ops_._linear_split(x, w, bias), torch.cat([torch.zeros(1, device=DEVICE), x.flatten()])[1:].view(m, k)
    torch.cuda.synchronize()
    ops_.raise_if_device_error()
    bound = (k / 64 + 48) * UNIT * (x.abs() @ w.abs().T + bias.abs())
    assert bool(((got.double() - (x.double() @ w.double().T + bias.double())).abs() <= bound.double()).all())
    # .. and in the 2-norm, where roundings average out: 1.1e-7 is what float32 itself gives; without the products of second and third parts 4e-6
    exact = x.double() @ w.double().T
    error, simt = ((t.double() - exact).norm(dim=1) / exact.norm(dim=1) for t in (ops_._linear_split(x, w, None),
                                                                                   ops_._linear_simt(x, w, None, torch.float32)))
    assert float(error.max()) <= 4e-7 and (k < 800 or float(error.mean()) <= float(simt.mean())), (float(error.max()), float(simt.mean()))
    assert torch.equal(ops_._linear_split(shifted, w, bias), got)          # x on no 16-byte boundary
    for first in {0, m // 2, m - 1}:
        assert torch.equal(ops_._linear_split(x[first:first + 1].contiguous(), w, bias), got[first:first + 1])
    if n % 128 == 0:
        gated = ops_.linear_swiglu(x, w, 64) if ops_._split_fits(x, w) else ops_._linear_split(x, w, None, gated=True)
        assert torch.equal(gated, ops_.swiglu(ops_._linear_split(x, w, None), 64))


@pytest.mark.parametrize("n,k", [(1152, 896), (9728, 100)])
def test_products_in_parts_with_infinities(n, k):
    """Infinities, NaN, zeros beside them, numbers at the ends of the range: what a chain of 32-bit multiply-adds makes of them."""
    x, w = rnd(1, 40, k), rnd(2, n, k, std=0.2)
    x[3, 5], x[4, 7], x[5, 9], x[6] = float("inf"), -float("inf"), float("nan"), 3.4e38
    w[10] = 0.0
    w[11, 5], w[12, 7], w[13, 0] = 1.0, float("inf"), float("nan")
    x[7], w[14] = 1e-38, 1e-3
    got, want = cuda()._linear_split(x.to(DEVICE), w.to(DEVICE), None).cpu(), cuda()._linear_simt(x.to(DEVICE), w.to(DEVICE), None, torch.float32).cpu()
    for kind in (torch.isnan, torch.isposinf, torch.isneginf):
        rows = torch.arange(40) != 6                 # of row 6 the order of the sum decides what overflows
        assert torch.equal(kind(got)[rows], kind(want)[rows])
    fine = torch.isfinite(got) & torch.isfinite(want)
    bound = (k + 48) * UNIT * (x.double().abs() @ w.double().abs().T) + k * 2.0 ** -134
    assert bool(((got.double() - want.double()).abs() <= bound)[fine].all())


def delta_inputs(rows, heads, kv_heads, dim, vdim, alike):
    """``alike``: keys that nearly repeat one another, steps near one, hardly any decay: the triangular systems at their hardest."""
    q, k, v = rnd(1, rows, kv_heads * dim), rnd(2, rows, kv_heads * dim), rnd(3, rows, heads * vdim)
    a, b, bias, a_log = rnd(4, rows, heads, std=2.0), rnd(5, rows, heads), rnd(6, heads), rnd(7, heads)
    if alike:
        k, a, b = k[:1] + 0.05 * k, a - 9.0, b + 6.0
    else:
        a[rows // 3], a[rows // 2], k[rows // 2 + 1] = 90.0, -90.0, 0.0      # all forgotten, nothing forgotten, no key at all
    return q, k, v, a, b, bias, a_log


@pytest.mark.parametrize("heads,kv_heads,dim,vdim", [(4, 2, 64, 64), (3, 1, 128, 48), (2, 2, 128, 80)])
@pytest.mark.parametrize("alike", [False, True])
@pytest.mark.parametrize("lengths,slots,order", CHUNKED)
def test_delta_rule_in_chunks(heads, kv_heads, dim, vdim, alike, lengths, slots, order, monkeypatch):
    """Segments around the borders of chunks, all of them in chunks or the short ones token by token beside."""
    ctx, rows = segments(lengths, slots, order), sum(lengths)
    q, k, v, a, b, bias, a_log = delta_inputs(rows, heads, kv_heads, dim, vdim, alike)
    state = rnd(8, len(lengths), heads, vdim, dim, std=0.3)
    want_state = state.double()
    want = FAKE.delta_rule_scan(*(t.double() for t in (q, k, v, a, b, bias, a_log)), want_state, ctx, heads, kv_heads, dim, vdim, 1e-6)
    for least in (1, 65, 128):
        monkeypatch.setattr(cuda(), "DELTA_CHUNK_ROWS", least)
        got_state = state.to(DEVICE)
        got = cuda().delta_rule_scan(*(spaced(t) for t in (q, k, v, a, b)), bias.to(DEVICE), a_log.to(DEVICE), got_state, ctx, heads,
                                     kv_heads, dim, vdim, 1e-6)
        # sums of up to dim + CHUNK products behind a triangular system of CHUNK rows
        close(got, want, 200 * UNIT, "delta rule outputs")
        close(got_state.flatten(0, 1), want_state.flatten(0, 1), 200 * UNIT, "delta rule state")


# 3.4e38: the largest bfloat16 number is below it
@pytest.mark.parametrize("value", [float("inf"), float("nan"), 3.4e38])
@pytest.mark.parametrize("which,at", [("k", 70), ("k", 110), ("v", 127), ("q", 199), ("a", 130), ("a", 105), ("b", 120)])
def test_a_token_that_is_no_number_leaves_the_tokens_of_a_delta_rule_before_it_alone(value, which, at, monkeypatch):
    monkeypatch.setattr(cuda(), "DELTA_CHUNK_ROWS", 64)
    heads, kv_heads, dim, vdim, rows = 2, 1, 128, 64, 200
    inputs = dict(zip("qkvab", delta_inputs(rows, heads, kv_heads, dim, vdim, False)))
    inputs["b"][at] = 90.0           # a value goes in whole
    bias, a_log = rnd(6, heads).to(DEVICE), rnd(7, heads).to(DEVICE)
    ctx, results = segments([rows], [0], None), []
    for broken in (False, True):
        given = {name: t.clone() for name, t in inputs.items()}
        if broken:
            given[which][at, 0] = value
        state = rnd(8, 1, heads, vdim, dim, std=0.3).to(DEVICE)
        results.append(cuda().delta_rule_scan(*(given[name].to(DEVICE) for name in "qkvab"), bias, a_log, state, ctx, heads, kv_heads, dim,
                                              vdim, 1e-6).cpu())
    assert torch.equal(results[0][:at], results[1][:at])


@pytest.mark.parametrize("heads,kv_heads,dim", [(8, 4, 128), (8, 4, 64)])
def test_delta_rule_in_chunks_is_no_further_from_64_bits(heads, kv_heads, dim, monkeypatch):
    """Inputs as behind a convolution's silu, whose keys have a common direction: the sums of their products grow, and with them what the
    tensor cores cut off.  The states' errors are sums of few roundings and differ from draw to draw, by a tenth in the mean of two."""
    vdim, rows = 64, 1024
    errors = {True: [0.0, 0.0], False: [0.0, 0.0]}
    for seed in (0, 20):
        silu = lambda index, width: torch.nn.functional.silu(rnd(seed + index, rows, width))      # noqa: E731
        inputs = (silu(1, kv_heads * dim), silu(2, kv_heads * dim), silu(3, heads * vdim), rnd(seed + 4, rows, heads), rnd(seed + 5, rows, heads),
                  torch.rand(heads, generator=generator(seed + 6)) * 4 - 4, torch.rand(heads, generator=generator(seed + 7)) * 2.5)
        ctx, want_state = segments([rows], [0]), torch.zeros(1, heads, vdim, dim, dtype=torch.float64)
        want = FAKE.delta_rule_scan(*(t.double() for t in inputs), want_state, ctx, heads, kv_heads, dim, vdim, 1e-6)
        for chunks in errors:
            monkeypatch.setattr(cuda(), "use_delta_chunks", chunks)
            state = torch.zeros(1, heads, vdim, dim, device=DEVICE)
            got = cuda().delta_rule_scan(*(t.to(DEVICE) for t in inputs), state, ctx, heads, kv_heads, dim, vdim, 1e-6)
            for index, (a, b) in enumerate(((got, want), (state, want_state))):
                errors[chunks][index] += float((a.double().cpu() - b).norm() / b.norm())
    assert errors[True][0] <= errors[False][0] and errors[True][1] <= 1.1 * errors[False][1], errors


def test_delta_rule_of_many_chunks_keeps_its_scratch_bounded():
    """More chunks than have their scratch in the bound: rounds of them, borders between rounds inside a portion and between portions."""
    heads, kv_heads, dim, vdim, lengths = 32, 16, 128, 64, [2700, 40, 600, 2300]
    ctx, rows = segments(lengths, [2, 0, 3, 1], [3, 1, 0, 2]), sum(lengths)
    q, k, v, a, b, bias, a_log = delta_inputs(rows, heads, kv_heads, dim, vdim, False)
    state = rnd(8, len(lengths), heads, vdim, dim, std=0.3)
    given, got_state = [t.to(DEVICE) for t in (q, k, v, a, b, bias, a_log)], state.to(DEVICE)
    torch.cuda.synchronize()
    torch.cuda.reset_peak_memory_stats()
    start = torch.cuda.memory_allocated()
    got = cuda().delta_rule_scan(*given, got_state, ctx, heads, kv_heads, dim, vdim, 1e-6)
    extra = torch.cuda.max_memory_allocated() - start - got.numel() * 4
    assert extra <= (257 << 20) + rows * heads * 48, extra      # and the inner products of the portions token by token
    want_state = state.to(DEVICE).double()
    want = FAKE.delta_rule_scan(*(t.double() for t in given), want_state, ctx, heads, kv_heads, dim, vdim, 1e-6)
    close(got, want.cpu(), 200 * UNIT, "delta rule outputs")
    close(got_state.flatten(0, 1), want_state.cpu().flatten(0, 1), 200 * UNIT, "delta rule state")


@pytest.mark.parametrize("known", [True, False])
@pytest.mark.parametrize("heads,kv_heads,dim,vdim", [(14, 7, 64, 64), (4, 1, 128, 32)])
def test_delta_rule_at_the_border_of_chunks(heads, kv_heads, dim, vdim, known, monkeypatch):
    """Portions on both sides of the border in one step, side by side; each has the bits of a step of its own.  ``known``: the lengths are on
    the host as well."""
    least, launched, load = cuda().DELTA_CHUNK_ROWS, [], cuda_ops.build.load_library
    lengths = [1, least - 1, least, 40, least + 65, 2, least - 30]
    ctx, rows = segments(lengths, [3, 0, 2, 1, 6, 5, 4], [4, 1, 6, 0, 5, 2, 3]), sum(lengths)
    parts = ctx.segments
    if not known:
        del ctx.segments
    q, k, v, a, b, bias, a_log = (t.to(DEVICE) for t in delta_inputs(rows, heads, kv_heads, dim, vdim, False))
    state = rnd(8, len(lengths), heads, vdim, dim, std=0.3)
    want_state = state.double()
    want = FAKE.delta_rule_scan(*(t.double().cpu() for t in (q, k, v, a, b, bias, a_log)), want_state, types.SimpleNamespace(
        seg_q_start=ctx.seg_q_start.cpu(), seg_q_len=ctx.seg_q_len.cpu(), seg_slot=ctx.seg_slot.cpu(), num_segments=len(lengths), segments=parts),
        heads, kv_heads, dim, vdim, 1e-6)
    monkeypatch.setattr(cuda_ops.build, "load_library", lambda name: launched.append(name) or load(name))
    for _ in range(3):
        launched.clear()
        got_state = state.to(DEVICE)
        got = cuda().delta_rule_scan(q, k, v, a, b, bias, a_log, got_state, ctx, heads, kv_heads, dim, vdim, 1e-6)
        following = got + got                   # behind both kernels' rows, those whose last launch it does not follow directly
        assert {"delta_rule", "delta_chunks"} <= set(launched)
        close(got, want, 200 * UNIT, "delta rule outputs")
        close(got_state.flatten(0, 1), want_state.flatten(0, 1), 200 * UNIT, "delta rule state")
        assert torch.equal(following, got * 2)
    graph, captured_state = torch.cuda.CUDAGraph(), state.to(DEVICE)
    torch.cuda.synchronize()
    with torch.cuda.graph(graph):
        captured = cuda().delta_rule_scan(q, k, v, a, b, bias, a_log, captured_state, ctx, heads, kv_heads, dim, vdim, 1e-6) * 2
    graph.replay()
    assert torch.equal(captured, following) and torch.equal(captured_state, got_state)
    for part in parts:
        at, own_state = slice(part.row_start, part.row_start + part.length), state.to(DEVICE)
        own = cuda().delta_rule_scan(*(t[at] for t in (q, k, v, a, b)), bias, a_log, own_state, segments([part.length], [part.slot]), heads,
                                     kv_heads, dim, vdim, 1e-6)
        if part.length > 1:                     # a decoded row is walked another way beside longer portions
            assert torch.equal(own, got[at]) and torch.equal(own_state[part.slot], got_state[part.slot]), part.length


@pytest.mark.parametrize("m,n,k", [(1, 8192, 2048), (40, 896, 4864), (300, 4864, 896)])
def test_products_in_parts_of_a_weight_just_written(m, n, k):
    """The product follows the kernel that writes its weight without anything between them."""
    x, base, step = (t.to(DEVICE) for t in (rnd(1, m, k), rnd(2, n, k, std=0.2), rnd(3, n, k, std=0.2)))
    assert cuda()._split_fits(x, base)
    want = cuda().linear(x, base + step)
    for _ in range(20):
        w = base.clone()
        assert torch.equal(cuda().linear(x, cuda().add_inplace(w, step)), want)


@pytest.mark.parametrize("n,k", [(1152, 896), (9728, 200), (896, 4864), (20100, 132), (33, 30000)])
@pytest.mark.parametrize("m", [1, 17, 40, 300])
def test_products_in_parts_whose_outputs_are_all_no_numbers(m, n, k):
    """Every output through the chains over k: values, and a time that is a batch's on the CUDA cores and not a thread's per output (a
    few microseconds per 64 k, where a CTA's steps over k follow one another)."""
    def timed(x):
        best = float("inf")
        for _ in range(3):
            start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            start.record()
            got = cuda()._linear_split(x, w, bias)
            end.record()
            torch.cuda.synchronize()
            best = min(best, start.elapsed_time(end))
        cuda().raise_if_device_error()
        return got, best

    x, w, bias = rnd(1, m, k).to(DEVICE), rnd(2, n, k, std=0.2).to(DEVICE), rnd(3, n).to(DEVICE)
    w[n // 2], w[n // 3, k - 1] = 0.0, -w[n // 3, k - 1]
    fine, plain = timed(x)
    broken = x.clone()
    broken[:, k - 1] = float("inf")
    got, took = timed(broken)
    assert torch.equal(torch.isnan(got), (w[:, k - 1] == 0).expand(m, n))
    assert torch.equal(got == float("inf"), (w[:, k - 1] > 0).expand(m, n)) and torch.equal(got == -float("inf"), (w[:, k - 1] < 0).expand(m, n))
    assert took <= 20 * plain + 0.1 + 1e-4 * k, (took, plain)
    if n % 128 == 0:
        assert torch.equal(cuda()._linear_split(broken, w, None, gated=True).nan_to_num(7.0),
                           cuda().swiglu(cuda()._linear_split(broken, w, None), 64).nan_to_num(7.0))
    broken.fill_(float("nan"))
    got, took = timed(broken)
    assert bool(torch.isnan(got).all()) and took <= 20 * plain + 0.1 + 1e-4 * k, (took, plain)
    x[m // 2, 0] = float("nan")                     # one row: the others keep their bits
    got, others = timed(x)[0], torch.arange(m, device=DEVICE) != m // 2
    assert bool(torch.isnan(got[m // 2]).all()) and torch.equal(got[others], fine[others])


def test_a_first_call_in_32_bits_may_be_captured():
    """A set of operations whose first calls are captured: no workspace is made inside a graph, where its counters would be zero only after
    a replay, and the products in bfloat16 that come next find theirs as they should be."""
    fresh = type(cuda())()
    x, w = rnd(1, 8, 896).to(DEVICE), rnd(2, 1152, 896, std=0.2).to(DEVICE)
    ctx, rows = segments([600], [0]), 600
    q, k, v, a, b, bias, a_log = (t.to(DEVICE) for t in delta_inputs(rows, 4, 2, 64, 64, False))
    state = torch.zeros(1, 4, 64, 64, device=DEVICE)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        product = fresh.linear(x, w)
        y = fresh.delta_rule_scan(q, k, v, a, b, bias, a_log, state, ctx, 4, 2, 64, 64, 1e-6)
    assert not fresh._workspaces
    rows = rnd(3, 64, 4864).to(DEVICE, torch.bfloat16), rnd(4, 896, 4864, std=0.02).to(DEVICE, torch.bfloat16)
    assert torch.equal(fresh.linear(*rows), cuda().linear(*rows))          # sums in parts, counted
    graph.replay()
    torch.cuda.synchronize()
    fresh.raise_if_device_error()
    assert torch.equal(product, cuda().linear(x, w))
    other = torch.zeros_like(state)
    assert torch.equal(y, cuda().delta_rule_scan(q, k, v, a, b, bias, a_log, other, ctx, 4, 2, 64, 64, 1e-6)) and torch.equal(state, other)


@pytest.mark.parametrize("lengths", [[576, 577, 640], [1088, 1089, 65], [2177]])
def test_states_carried_over_many_chunks(lengths):
    """Segments around the numbers of chunks that the carrying kernels ask for at a time: one turn, two and three."""
    ctx, rows, heads, n = segments(lengths, list(reversed(range(len(lengths)))), None), sum(lengths), 3, 64
    inner, bound = heads * 64, 200 * UNIT
    x, B, C, dt = rnd(1, rows, inner), rnd(2, rows, n), rnd(3, rows, n), rnd(4, rows, heads, std=2.0)
    vectors = rnd(5, heads), rnd(6, heads), rnd(7, heads)
    state = rnd(8, len(lengths), heads, 64, n, std=0.5)
    want_state, got_state = state.double(), state.to(DEVICE)
    want = FAKE.state_space_scan(*(t.double() for t in (x, B, C, dt, *vectors)), want_state, ctx, heads, 64, n, 1)
    got = cuda().state_space_scan(*(spaced(t) for t in (x, B, C, dt)), *(t.to(DEVICE) for t in vectors), got_state, ctx, heads, 64, n, 1)
    close(got, want, bound, "state-space outputs")
    close(got_state.flatten(0, 1), want_state.flatten(0, 1), bound, "state-space state")
    r, k, v, gate, raw = (rnd(10 + i, rows, inner, std=0.7) for i in range(5))
    bias, bonus, weight = rnd(16, inner) * 2 - 2, rnd(17, inner, std=0.3), 1 + rnd(18, inner, std=0.1)
    want_state, got_state = state.double(), state.to(DEVICE)
    want = FAKE.bonus_recurrence(*(t.double() for t in (r, k, v, raw, gate, bias, bonus, weight)), 1e-6, want_state, ctx, heads, 64, torch.float32)
    got = cuda().bonus_recurrence(*(spaced(t) for t in (r, k, v, raw, gate)), *(t.to(DEVICE) for t in (bias, bonus, weight)), 1e-6, got_state, ctx,
                                  heads, 64, torch.float32)
    close(got, want, bound, "recurrence outputs")
    close(got_state.flatten(0, 1), want_state.flatten(0, 1), bound, "recurrence state")


@pytest.mark.parametrize("m", [9, 27, 60, 200])
@pytest.mark.parametrize("places", [(0, 1, 2), (3, 40, 17), (63, 64, 895), (500, 130, 129)])
def test_products_in_parts_take_each_product_of_parts(m, places):
    """Numbers of one to three parts (1, 2^-9 and 2^-18 beside it) whose leading products cancel, so that what is left is one product of
    smaller parts; those left out are 2^-27 and less, every sum is exact."""
    n, k, (a, b, c) = 1152, 896, places
    x, w = torch.zeros(m, k), torch.zeros(n, k)
    numbers = torch.tensor([1.0, 1 + 2.0 ** -18, 1 + 2.0 ** -9, 1 + 2.0 ** -9 + 2.0 ** -18])
    x[:, a], x[:, b], x[:, c] = numbers[torch.arange(m) % 4], -1.0, torch.where(torch.arange(m) % 3 == 0, -2.0 ** -8, 0.0)
    w[:, a], w[:, b], w[:, c] = numbers[torch.arange(n) % 4], 1.0, 1.0
    got, want = cuda()._linear_split(x.to(DEVICE), w.to(DEVICE), None).double().cpu(), x.double() @ w.double().T
    assert float((got - want).abs().max()) <= 3 * 2.0 ** -27


@pytest.mark.parametrize("m,n,k,gated", [(641, 33, 30000, False), (1300, 33, 30000, False), (672, 256, 30000, True)])
def test_products_in_parts_of_rows_in_blocks(m, n, k, gated):
    """More rows than have their parts in scratch at a time (640 of 30,000 k): blocks of rows with the bits of calls of their own, the last of one
    row, of 20 and of 32."""
    x, w, bias = (t.to(DEVICE) for t in (rnd(1, m, k), rnd(2, n, k, std=0.02), rnd(3, n)))
    product = lambda rows: cuda()._linear_split(rows, w, None if gated else bias, gated=gated)      # noqa: E731
    torch.cuda.synchronize()
    torch.cuda.reset_peak_memory_stats()
    start = torch.cuda.memory_allocated()
    whole = product(x)
    extra = torch.cuda.max_memory_allocated() - start - whole.numel() * 4
    assert extra <= 129 << 20, extra
    exact = x.double() @ w.double().T
    if gated:
        gate, up = exact.view(m, -1, 2, 64).unbind(2)
        exact = (torch.nn.functional.silu(gate) * up).reshape(m, -1)
    else:
        exact += bias.double()
    assert float((whole.double() - exact).norm() / exact.norm()) <= 1e-6
    for first, rows in ((0, 640), (640, min(m, 1280) - 640), (m - 1, 1), (m - 20, 20), (630, 11)):
        assert torch.equal(product(x[first:first + rows].contiguous()), whole[first:first + rows]), first


@pytest.mark.parametrize("n,k", [(16400, 73), (3000, 4101)])
def test_products_that_the_tensor_cores_do_not_take(n, k):
    """Rows of no whole 16-byte pieces: the product on the CUDA cores, more than 16,384 outputs, long sums in parts of many rows in blocks."""
    m = 4000 if k > 4000 else 300
    x, w, bias = (t.to(DEVICE) for t in (rnd(1, m, k), rnd(2, n, k, std=0.2), rnd(3, n)))
    assert not cuda()._split_fits(x, w)
    torch.cuda.synchronize()
    torch.cuda.reset_peak_memory_stats()
    start = torch.cuda.memory_allocated()
    whole = cuda().linear(x, w, bias)
    extra = torch.cuda.max_memory_allocated() - start - whole.numel() * 4
    assert extra <= 129 << 20, extra
    for first, rows in ((0, 64), (m // 3, 100), (m - 63, 63), (m - 1, 1)):
        exact = x[first:first + rows].double() @ w.double().T + bias.double()
        assert bool(((whole[first:first + rows].double() - exact).abs()
                     <= k * UNIT * (x[first:first + rows].abs() @ w.abs().T + bias.abs()).double()).all())
        assert torch.equal(cuda().linear(x[first:first + rows].contiguous(), w, bias), whole[first:first + rows]), first
