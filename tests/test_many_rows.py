"""The kernels of steps with many rows, at the sizes where their tiles, remainders and runs can go
wrong, against float64 statements and against the kernels for few rows."""
import pytest
import torch

from llmario_b200.kernels import recurrence_runs, recurrence_work_floats

gpu = pytest.mark.gpu
DEV = "cuda:0"


def rnd(*shape, dtype=torch.float32, scale=1.0, seed=0):
    g = torch.Generator().manual_seed(seed + sum(shape))
    return (scale * torch.randn(*shape, generator=g)).to(dtype).to(DEV)


@gpu
@pytest.mark.parametrize("accumulate", [False, True])
@pytest.mark.parametrize("M,N,K,pad", [(1, 130, 128, 0), (16, 1024, 2048, 4), (17, 33, 1028, 0), (32, 64, 20, 8),
                                       (40, 72, 36, 0), (33, 257, 256, 0), (64, 128, 260, 0), (70, 96, 4, 0),
                                       (95, 128, 1024, 0), (129, 1000, 1040, 0), (211, 1024, 3072, 0),
                                       (130, 16500, 64, 0)])
def test_gemm_float32(M, N, K, pad, accumulate):
    """Tiles of 16 and of 32 to 64 rows, K whole and in parts, ragged N, K below one step, padded
    rows; a row's bits do not depend on how many rows there are."""
    from llmario_b200 import kernels
    a, w = rnd(M, K + pad, seed=1)[:, :K], rnd(N, K + pad, seed=2)[:, :K]
    c0 = rnd(M, N, seed=3)
    out = c0.clone()
    kernels.gemm_simt(a, w, out, accumulate)
    ref = a.double() @ w.double().T + (c0.double() if accumulate else 0)
    # every partial sum is rounded once per addition: |error| <= (K + 10) 2^-24 sum |a w|, and far
    # less on average
    size = a.abs().double() @ w.abs().double().T + (c0.abs().double() if accumulate else 0)
    assert bool(((out.double() - ref).abs() <= (K + 10) * 2 ** -24 * size).all())
    rel = float((out.double() - ref).norm() / ref.norm())
    assert rel <= 2 ** -24 * (2 + K ** 0.5)      # roundings that do not conspire
    for rows in (1, 17, 40):
        if rows < M:
            few = c0[:rows].clone()
            kernels.gemm_simt(a[:rows], w, few, accumulate)
            assert torch.equal(few, out[:rows])


def test_runs_cover_the_rows_and_fit_their_work():
    for rows in (1, 100, 255, 256, 383, 384, 1000, 1023, 1024, 2048, 8191):
        for H, K, V in ((4, 128, 256), (32, 128, 64), (1, 30, 7), (16, 250, 33), (16, 128, 256), (128, 128, 64)):
            parts, run = recurrence_runs(rows, H, K, V)
            floats = recurrence_work_floats([rows, 1, 1], H, K, V)
            if parts == 1:
                assert floats == 0
            else:
                assert parts * run >= rows and (parts - 1) * run < rows and run % 16 == 0 and parts <= 32
                assert floats == parts * H * (V + 1) * K and floats < 2 ** 27
                assert recurrence_work_floats([rows, rows, 3], H, K, V) == 2 * floats
    assert recurrence_runs(2048, 128, 128, 64) == (1, 0) and recurrence_runs(300, 4, 128, 256)[0] > 1


@gpu
@pytest.mark.parametrize("H,G,K,V,lengths", [(2, 1, 128, 64, [2048]), (4, 4, 128, 256, [257]), (3, 3, 30, 7, [500, 3, 1, 290]),
                                             (2, 2, 72, 20, [96, 480]), (1, 1, 256, 16, [320, 64]),
                                             (2, 1, 200, 40, [288, 111]),
                                             (1, 1, 8, 4, [1, 260] + [1] * 40 + [2, 511, 256, 255] + [3] * 30 + [777])])
@pytest.mark.parametrize("kind", (0, 1, 2, 3))
def test_recurrence_in_runs(kind, H, G, K, V, lengths):
    """Long portions in runs against the formula in float64 and against the whole walk, states that
    carry on from an earlier step, requests that end in their first run."""
    from llmario_b200 import kernels
    if kind in (0, 1) and G != H:
        G = H
    rows, n_slots = sum(lengths), len(lengths) + 2
    assert recurrence_runs(max(lengths), H, K, V)[0] > 1
    slots = list(range(n_slots - 1, n_slots - 1 - len(lengths), -1))
    row_slot = torch.tensor(sum(([s] * n for s, n in zip(slots, lengths)), []), dtype=torch.int32, device=DEV)
    seg = torch.empty(n_slots, 3, dtype=torch.int32, device=DEV)
    kernels.segment_table(row_slot, seg)
    q, k, v = rnd(rows, G * K, seed=1), rnd(rows, G * K, seed=2, scale=0.3), rnd(rows, H * V - (H if kind == 3 else 0), seed=3)
    d = rnd(rows, H if kind >= 2 else H * K, seed=4) + 2
    d2 = None
    if kind in (0, 3):
        d = torch.sigmoid(d + 2)
    if kind == 3:
        d2 = rnd(rows, H, seed=5).abs()
    p0, p1 = rnd(H, seed=6) - 2, rnd(H, seed=7)
    start = rnd(n_slots, H * V * K + 3, seed=8)

    def go(work):
        state = start.clone()
        out = torch.full((rows, H * V), float("nan"), device=DEV)
        kernels.linear_recurrence(q, k, v, d, state, out, row_slot, seg, H, G, K, V, kind, q_scale=0.5, exponent=0.25,
                                  rate_log=p0, step_bias=p1, n_requests=len(lengths), input_weight=d2, ones=kind == 3,
                                  work=work, portions=lengths)
        return state, out

    work = torch.full((recurrence_work_floats(lengths, H, K, V),), float("nan"), device=DEV)
    state, out = go(work)
    state_w, out_w = go(None)
    S = start[:, :H * V * K].double().view(n_slots, H, V, K).clone()
    ref = torch.zeros(rows, H, V, dtype=torch.float64, device=DEV)
    vd = v.double().view(rows, H, -1)
    if kind == 3:
        vd = torch.cat([vd, torch.ones(rows, H, 1, dtype=torch.float64, device=DEV)], -1) * d2.double()[..., None]
    if kind == 2:
        dt = torch.nn.functional.softplus(d.double() + p1.double())
        a = torch.exp(-torch.exp(p0.double()) * dt)[..., None].expand(rows, H, K)
        vd = vd * dt[..., None]
    elif kind == 3:
        a = d.double()[..., None].expand(rows, H, K)
    else:
        a = d.double().view(rows, H, K)
        if kind == 1:
            a = torch.sigmoid(a) ** 0.25
    kd = k.double().view(rows, G, K).repeat_interleave(H // G, 1)
    qd = 0.5 * q.double().view(rows, G, K).repeat_interleave(H // G, 1)
    r = 0
    for s, n in zip(slots, lengths):
        for _ in range(n):
            S[s] = S[s] * a[r][:, None, :] + vd[r][:, :, None] * kd[r][:, None, :]
            ref[r] = (S[s] * qd[r][:, None, :]).sum(-1)
            r += 1
    err = lambda x, y: float((x.double() - y).norm() / y.norm())  # noqa: E731
    e_out, e_whole = err(out, ref.view(rows, -1)), err(out_w, ref.view(rows, -1))
    got, whole = (t[:, :H * V * K].reshape(S.shape) for t in (state, state_w))
    # A state gets one rounding more per run (the carry's) among those of hundreds of tokens: the runs are
    # no further off than the whole walk, but for a quarter of a rounding in the norm
    assert e_out <= e_whole + 2 ** -26 and err(got, S) <= err(whole, S) + 2 ** -26 and e_out < 1e-6
    assert torch.equal(state[:, H * V * K:], start[:, H * V * K:])
    assert torch.equal(state[:2], start[:2])                  # slots without rows


@gpu
@pytest.mark.parametrize("H,K,V,lengths", [(4, 128, 256, [600, 1, 1, 255, 3, 256]), (32, 128, 64, [1, 2, 500, 384, 383]),
                                           (16, 128, 256, [1, 1100]), (3, 30, 7, [300, 1, 256])])
@pytest.mark.parametrize("kind", (0, 2))
def test_a_request_gives_the_same_bits_alone_and_in_company(kind, H, K, V, lengths):
    """Whether a portion goes in runs, and where it is cut, is its own: decoded tokens and short portions
    beside long ones, and long ones beside others, give the bits that they give alone."""
    from llmario_b200 import kernels
    rows = sum(lengths)
    q, k, v = rnd(rows, H * K, seed=1), rnd(rows, H * K, seed=2, scale=0.3), rnd(rows, H * V, seed=3)
    d = torch.sigmoid(rnd(rows, H * K, seed=4) + 4) if kind == 0 else rnd(rows, H, seed=4)
    p0, p1 = rnd(H, seed=6) - 2, rnd(H, seed=7)
    start = rnd(len(lengths), H * V * K, seed=8)

    def go(which):
        at = [sum(lengths[:i]) for i in range(len(lengths))]
        pick = sum((list(range(at[i], at[i] + lengths[i])) for i in which), [])
        mine = [lengths[i] for i in which]
        row_slot = torch.tensor(sum(([i] * lengths[i] for i in which), []), dtype=torch.int32, device=DEV)
        seg = None
        if any(n > 1 for n in mine):
            seg = torch.empty(len(lengths), 3, dtype=torch.int32, device=DEV)
            kernels.segment_table(row_slot, seg)
        state, out = start.clone(), torch.full((len(pick), H * V), float("nan"), device=DEV)
        work = torch.full((recurrence_work_floats(mine, H, K, V),), float("nan"), device=DEV)
        kernels.linear_recurrence(q[pick], k[pick], v[pick], d[pick], state, out, row_slot, seg, H, H, K, V, kind,
                                  q_scale=0.5, rate_log=p0, step_bias=p1, n_requests=len(which),
                                  work=work if len(work) else None, portions=mine)
        return state, out

    state, out = go(range(len(lengths)))
    for i, n in enumerate(lengths):
        state_i, out_i = go([i])
        at = sum(lengths[:i])
        assert torch.equal(out_i, out[at:at + n]), (i, n)
        assert torch.equal(state_i[i], state[i]), (i, n)


@gpu
@pytest.mark.parametrize("T,N,K", [(777, 4096, 1024), (1024, 520, 72), (543, 6144, 200), (2048, 1024, 3072),
                                   (513, 264, 512), (586, 8200, 3080), (1500, 136, 4096), (600, 4096, 2056), (2049, 520, 1024)])
def test_linear_many_rows_few_tiles(T, N, K):
    """Products with fewer tiles than CTAs, stored whole or added in ranges of K."""
    from llmario_b200 import kernels
    a, w = rnd(T, K, dtype=torch.bfloat16, seed=1), rnd(N, K, dtype=torch.bfloat16, seed=2)
    wide = torch.full((T, N + 8), float("nan"), device=DEV)
    kernels.linear(a, w, wide[:, :N])
    ref = a.double() @ w.double().T
    # 32-bit sums of exact products of 16-bit operands
    bound = (K + 10) * 2 ** -23 * (a.abs().double() @ w.abs().double().T)
    assert bool(((wide[:, :N].double() - ref).abs() <= bound).all())
    assert bool(torch.isnan(wide[:, N:]).all())
    kernels.check_tc_status(torch.device(DEV))


@gpu
@pytest.mark.parametrize("group,hd,window,page", [(1, 64, 0, 16), (2, 128, 0, 64), (4, 128, 50, 16), (8, 64, 33, 4),
                                                  (2, 64, -48, 32), (8, 128, 0, 8)])
def test_attention_float32_tiles_give_the_bits_of_single_rows(group, hd, window, page):
    """Blocks of consecutive tokens go by tiles, the rest row by row: both give the same bits,
    whatever is in the step (a request's end inside a block, single tokens between portions, values
    that are not finite at positions a row does not see)."""
    from llmario_b200 import kernels
    Hkv = 2
    Hq = Hkv * group
    segments = [(0, 37), (900, 1), (5, 70), (3, 3), (64, 16), (0, 1), (31, 45)]      # (first position, rows)
    slots = [4, 0, 6, 1, 3, 2, 5]
    n_pages = sum(-(-(p + n) // page) for p, n in segments)
    storage = rnd(n_pages, 2, Hkv, page, hd, seed=5)
    table = torch.full((7, 1024 // page), -1, dtype=torch.int32)
    used = 0
    row_slot, row_pos = [], []
    for (p, n), slot in zip(segments, slots):
        need = -(-(p + n) // page)
        table[slot, :need] = torch.randperm(need, generator=torch.Generator().manual_seed(slot)).int() + used
        used += need
        row_slot += [slot] * n
        row_pos += list(range(p, p + n))
    # the last position of the first request holds values that no other row may meet
    last = segments[0][1] - 1
    storage[int(table[4, last // page]), 1, :, last % page] = float("inf")
    rs = torch.tensor(row_slot, dtype=torch.int32, device=DEV)
    rp = torch.tensor(row_pos, dtype=torch.int32, device=DEV)
    table = table.to(DEV)
    q = rnd(len(row_slot), Hq * hd, seed=7)

    def run(rows):
        out = torch.full((len(rows), Hq * hd), float("nan"), device=DEV)
        kernels.attention_generic(q[rows].contiguous(), out, storage[:, 0], storage[:, 1], storage.stride(0), table,
                                  rs[rows].contiguous(), rp[rows].contiguous(), Hq, Hkv, hd, page, hd ** -0.5, window)
        return out

    everything = run(list(range(len(row_slot))))
    # eight rows are fewer than a block: row by row
    alone = torch.cat([run(list(range(i, min(i + 8, len(row_slot))))) for i in range(0, len(row_slot), 8)])
    finite = [i for i in range(len(row_slot)) if i != last]
    assert bool(torch.isfinite(everything[finite]).all())
    assert torch.equal(everything[finite], alone[finite])


def test_uniforms_of_many_streams():
    """The native draw: every stream's own next number, in order, nothing for streams left out."""
    import ctypes
    from llmario_b200.sampling.rng import Xoshiro256StarStar, next_uniforms
    mine, alone = ([Xoshiro256StarStar(s) for s in (0, 1, 2 ** 64 - 1, 7)] for _ in range(2))
    out = (ctypes.c_double * 5)(*[9.0] * 5)
    for _ in range(3):
        next_uniforms([mine[0], None, mine[1], mine[2], mine[0]], ctypes.addressof(out))
        assert list(out) == [alone[0].next_f64(), 0.0, alone[1].next_f64(), alone[2].next_f64(), alone[0].next_f64()]
    assert mine[3].next_u64() == alone[3].next_u64()


def test_a_stream_is_saved_restored_and_copied():
    """A request's sampling state goes through pickle in the middle of its stream, as its four numbers
    do through JSON; the numbers may be set, or changed in place; what earlier versions saved is read."""
    import copy
    import ctypes
    import json
    import pickle
    from llmario_b200.sampling import RequestSampler, SamplingParams
    from llmario_b200.sampling.rng import Xoshiro256StarStar, next_uniforms
    a = RequestSampler(SamplingParams(seed=3), 100)
    a.next_uniform()
    b = pickle.loads(pickle.dumps(a))
    c, text = copy.deepcopy(a), json.dumps(a.rng.s)
    d = Xoshiro256StarStar(99)
    d.s = json.loads(text)
    old = Xoshiro256StarStar.__new__(Xoshiro256StarStar)
    old.__setstate__({"s": json.loads(text)})
    e = Xoshiro256StarStar(0)
    e.s[:] = json.loads(text)
    assert isinstance(a.rng.s, list) and d.s == a.rng.s == e.s

    class Twice(Xoshiro256StarStar):
        def next_f64(self):
            return super().next_f64() / 2

    half, plain = Twice(3), Xoshiro256StarStar(3)
    half.next_u64(), plain.next_u64()
    out = (ctypes.c_double * 7)()
    for _ in range(3):
        next_uniforms([a.rng, b.rng, c.rng, d, old, e, half], ctypes.addressof(out))
        want = plain.next_f64()
        assert list(out) == [want] * 6 + [want / 2]
    assert a.rng.s == d.s == plain.s and a.rng.next_u64() == plain.next_u64()
    shared = copy.copy(plain)                    # a shallow copy is the same stream
    first = plain.next_u64()
    assert shared.next_u64() != first and shared.s is plain.s


@gpu
@pytest.mark.parametrize("bn", (32, 64, 128))
@pytest.mark.parametrize("counts,N,K", [([300, 0, 1, 129, 256, 64], 512, 256), ([700, 33, 32], 272, 72),
                                        ([0, 0, 5], 96, 200), ([64] * 40, 64, 64)])
def test_grouped_products_on_cta_pairs(counts, N, K, bn):
    """Tiles of one matrix joined to as many as 256 rows, matrices without rows, ragged N and K, every
    epilogue; padding rows hold NaN and rows of matrices without tiles are not written."""
    from llmario_b200 import kernels
    E = len(counts)
    tiles = [-(-c // bn) for c in counts]
    T = (sum(tiles) + 2) * bn                       # two tiles that are left out
    x = torch.full((T, K), float("nan"), dtype=torch.bfloat16, device=DEV)
    group, rows, expert = [], [], []
    for e, c in enumerate(counts):
        rows += range(len(group) * bn, len(group) * bn + c)
        expert += [e] * c
        group += [e] * tiles[e]
    x[rows] = rnd(len(rows), K, dtype=torch.bfloat16, seed=1)
    tg = torch.tensor(group + [-1, -1], dtype=torch.int32, device=DEV)
    w = rnd(E, N, K, dtype=torch.bfloat16, seed=2, scale=K ** -0.5)
    scale = torch.full((T,), float("nan"), device=DEV)
    scale[rows] = rnd(len(rows), seed=3).abs()
    ex = torch.tensor(expert, device=DEV)
    xr = x[rows].double()
    ref = torch.zeros(len(rows), N, dtype=torch.float64, device=DEV)
    size = torch.zeros_like(ref)
    for e in range(E):
        ref[ex == e] = xr[ex == e] @ w[e].double().T
        size[ex == e] = xr[ex == e].abs() @ w[e].abs().double().T
    out = torch.full((T, N), 7.0, device=DEV)
    kernels.gemm_grouped(x, w, out, tg, bn, gated=False, paired=True)
    assert bool(((out[rows].double() - ref).abs() <= (K + 10) * 2 ** -23 * size).all())
    assert bool((out[sum(tiles) * bn:] == 7.0).all())
    r2 = torch.full((T, N), 7.0, dtype=torch.bfloat16, device=DEV)
    kernels.gemm_grouped(x, w, r2, tg, bn, gated=False, activation="relu_squared", paired=True)
    want = ref.clamp(min=0) ** 2
    # 32-bit sums, squared, rounded to 8 bits of mantissa
    assert bool(((r2[rows].double() - want).abs() <= 2 ** -8 * want + (K + 10) * 2 ** -21 * size * (size + 1)).all())
    kernels.check_tc_status(torch.device(DEV))
    if N % 32:
        return
    half = N // 2
    blocks = ref.view(len(rows), N // 32, 2, 16)
    gate, up = blocks[:, :, 0].reshape(-1, half), blocks[:, :, 1].reshape(-1, half)
    act = torch.full((T, half), 7.0, dtype=torch.bfloat16, device=DEV)
    one = torch.empty(T, half, dtype=torch.bfloat16, device=DEV)
    for kw in (dict(), dict(activation="clamped_swish", limit=0.8, row_scale=scale)):
        kernels.gemm_grouped(x, w, act, tg, bn, gated=True, interleaved=True, paired=True, **kw)
        kernels.gemm_grouped(x, w, one, tg, bn, gated=True, interleaved=True, **kw)
        if kw:
            s = scale[rows].double()[:, None]
            g, u = (gate * s).clamp(max=0.8), (up * s).clamp(-0.8, 0.8)
            want = g * torch.sigmoid(1.702 * g) * (u + 1)
        else:
            want = gate * torch.sigmoid(gate) * up
        # rounding of the result, and of 32-bit sums in front of functions with slopes below 2
        bound = 2 ** -8 * want.abs() + 1e-5 * (1 + want.abs())
        assert bool(((act[rows].double() - want).abs() <= bound).all())
        assert torch.equal(act[rows], one[rows])       # the same sums in the same order
        assert bool((act[sum(tiles) * bn:] == 7.0).all())
    kernels.check_tc_status(torch.device(DEV))


@gpu
@pytest.mark.parametrize("rows", (1, 2, 3, 4))
@pytest.mark.parametrize("N,K", [(1024, 2048), (4096, 1024), (1024, 3072), (148, 1024), (7, 2048), (3056, 1024), (640, 256),
                                 (96, 4096), (200, 768), (1000, 1536), (300, 2304), (3600, 2048)])
def test_row_product(rows, N, K):
    """One to four rows through a small matrix (held in registers or in shared memory): stored, added,
    gated, of 16-bit rows and of the norm of 32-bit rows; fewer outputs than SMs, slices that do not
    come out even, strided rows."""
    from llmario_b200 import kernels
    if (N, K) == (3600, 2048) and rows > 2:      # (slices of 100 KB: no room for more rows beside them)
        assert not kernels.row_product_ok(rows, N, K)
        return
    assert kernels.row_product_ok(rows, N, K)
    x = rnd(rows, K + 8, seed=1)[:, :K]
    h = rnd(rows, K + 8, dtype=torch.bfloat16, seed=2)[:, :K]
    g = 1 + 0.1 * rnd(K, seed=3)
    w = rnd(N, K, dtype=torch.bfloat16, seed=4, scale=K ** -0.5)
    xd = x.double()
    normed = (xd * torch.rsqrt((xd * xd).mean(-1, keepdim=True) + 1e-6) * g.double())
    out = torch.full((rows, N + 4), float("nan"), device=DEV)
    for src, kw, exact in ((h, {}, h.double()), (x, dict(norm_weight=g, eps=1e-6), normed)):
        ref = exact @ w.double().T
        size = exact.abs() @ w.double().abs().T
        # 32-bit sums; a normed row is rounded to 8 bits of mantissa first, each value by up to 2^-9
        bound = (K + 10) * 2 ** -23 * size + (2 ** -9 * size if kw else 0)
        kernels.row_product(src, w, out[:, :N], **kw)
        assert bool(((out[:, :N].double() - ref).abs() <= bound).all())
        first = out[:, :N].clone()
        kernels.row_product(src, w, out[:, :N], accumulate=True, **kw)
        assert torch.equal(out[:, :N], first + first)
        assert bool(torch.isnan(out[:, N:]).all())
        if N % 32 == 0 and kernels.row_product_ok(rows, N // 2, K, True):
            act = torch.empty(rows, N // 2, dtype=torch.bfloat16, device=DEV)
            kernels.row_product(src, w, act, gated=True, **kw)
            b = ref.view(rows, N // 32, 2, 16)
            gate, up = b[:, :, 0].reshape(rows, -1), b[:, :, 1].reshape(rows, -1)
            want = gate * torch.sigmoid(gate) * up
            s = size.view(rows, N // 32, 2, 16).amax(2).reshape(rows, -1) if kw else 0
            slack = 2 ** -9 * s * (2 + gate.abs() + up.abs()) if kw else 0
            assert bool(((act.double() - want).abs() <= 2 ** -8 * want.abs() + 1e-5 * (1 + want.abs()) + slack).all())
    kernels.check_tc_status(torch.device(DEV))


@gpu
@pytest.mark.parametrize("T,N,K", [(1501, 4096, 4096), (700, 6144, 1096), (520, 6144, 4096), (2048, 2304, 2056), (900, 4096, 584),
                                   (1024, 4608, 520)])
def test_linear_in_two_ranges_keeps_its_sum(T, N, K):
    """A product that is asked for in two ranges of K is their sum, whichever kernel makes it (odd
    numbers of blocks of K, ragged N, last tokens)."""
    from llmario_b200 import kernels
    assert kernels.k_splits(T, N, K) == 2
    a, w = rnd(T, K, dtype=torch.bfloat16, seed=1), rnd(N, K, dtype=torch.bfloat16, seed=2)
    got, lone = torch.empty(T, N, device=DEV), torch.empty(T, N, device=DEV)
    kernels.linear(a, w, got)
    kernels.use_cta_pairs(False)
    try:
        kernels.linear(a, w, lone)
    finally:
        kernels.use_cta_pairs(True)
    assert torch.equal(got, lone)
    got.zero_()
    kernels.linear(a, w, got, out_is_zero=True)
    assert torch.equal(got, lone)
    kernels.check_tc_status(torch.device(DEV))


@gpu
@pytest.mark.parametrize("T,N,K", [(513, 4096, 1024), (545, 6144, 3072), (600, 5120, 4096)])
def test_added_products_stay_whole_with_few_last_tokens(T, N, K):
    """Where whole tiles are summed over K at once, so are tiles beside a narrow one."""
    from llmario_b200 import kernels
    a, w = rnd(T, K, dtype=torch.bfloat16, seed=1), rnd(N, K, dtype=torch.bfloat16, seed=2)
    got = rnd(T, N, seed=3)
    whole = got.clone()
    kernels.linear(a, w, got, accumulate=True)
    kernels.force_pair_k_ranges(1)
    try:
        kernels.linear(a, w, whole, accumulate=True)
    finally:
        kernels.force_pair_k_ranges(0)
    assert torch.equal(got, whole)
    kernels.check_tc_status(torch.device(DEV))


@gpu
@pytest.mark.parametrize("rows", (1, 3))
def test_linear_takes_wider_operands_at_few_rows(rows):
    """A matrix with more columns than the rows have, and an output with more rows and columns than
    the product: the leading part is what is used, whatever the number of rows."""
    from llmario_b200 import kernels
    a = rnd(rows, 1024, dtype=torch.bfloat16, seed=1)
    w = rnd(96, 1280, dtype=torch.bfloat16, seed=2)
    out = torch.zeros(rows + 2, 128, device=DEV)
    kernels.linear(a, w, out)
    ref = a.double() @ w[:, :1024].double().T
    bound = (1024 + 10) * 2 ** -23 * (a.abs().double() @ w[:, :1024].abs().double().T)
    assert bool(((out[:rows, :96].double() - ref).abs() <= bound).all())
    assert not out[rows:].any() and not out[:, 96:].any()
    kernels.check_tc_status(torch.device(DEV))


@gpu
@pytest.mark.parametrize("T,N,K,splits", [(1, 16384, 512, 2), (8, 16388, 512, 2), (3, 1028, 1024, 4), (40, 4096, 512, 2),
                                          (1300, 512, 512, 2)])
def test_the_output_of_a_cut_product_is_cleared_first(T, N, K, splits):
    """Few wide rows in pieces, many rows in turn, columns that are not whole pieces; nothing beside the
    output is touched."""
    from llmario_b200 import kernels
    a, w = rnd(T, K, dtype=torch.bfloat16, seed=1), rnd(N, K, dtype=torch.bfloat16, seed=2)
    wide = torch.full((T, N + 8), 7.0, device=DEV)
    kernels.gemm_tcgen05(a, w, wide[:, :N], 0, splits=splits, bn=64)
    ref = a.double() @ w.double().T
    bound = (K + 10) * 2 ** -23 * (a.abs().double() @ w.abs().double().T)
    assert bool(((wide[:, :N].double() - ref).abs() <= bound).all())
    assert bool((wide[:, N:] == 7.0).all())
    kernels.check_tc_status(torch.device(DEV))


@gpu
def test_the_choice_of_pairs_knows_when_they_are_off():
    """A product of many rows is not prepared for CTA pairs that will not run: its output is then
    cleared only where the lone CTAs add into it."""
    from llmario_b200 import kernels
    way = kernels.lib().llm_pair_store_way
    sizes = [(777, 4096, 1024, 2), (2048, 1024, 3072, 5), (1501, 4096, 4096, 2), (513, 1024, 1024, 4)]
    assert [way(*s) for s in sizes] == [0, 1, 1, 2]
    kernels.use_cta_pairs(False)
    try:
        assert [way(*s) for s in sizes] == [2] * 4
    finally:
        kernels.use_cta_pairs(True)


@gpu
def test_launches_of_the_generic_attention_are_counted():
    """A prompt in 32-bit takes two kernels per layer, as many decoded tokens one, and the counts say so."""
    from llmario_b200 import Model, ModelRunner, StepEntry, driver, kernels
    from llmario_b200.config import Qwen3Config
    from llmario_b200.weights import random_tensors
    cfg = Qwen3Config.from_dict(dict(
        architectures=["Qwen3ForCausalLM"], model_type="qwen3", max_position_embeddings=512, num_hidden_layers=3,
        hidden_size=64, num_attention_heads=4, num_key_value_heads=2, head_dim=64, intermediate_size=128,
        vocab_size=256, rope_theta=10000.0, rms_norm_eps=1e-6, tie_word_embeddings=True, torch_dtype="float32"))
    spec = cfg.to_spec()
    model = Model(spec, random_tensors(spec, 1, torch.float32, DEV), torch.float32, DEV)
    runner = ModelRunner(model, page_size=16, n_pages=64, max_requests=20, max_context=64, use_graphs=False)

    def counted(entries):
        runner.step(entries)
        torch.cuda.synchronize()
        with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
            was, generic = kernels.launches, driver.kernel_counts()["generic"]
            runner.step(entries)
            torch.cuda.synchronize()
            said = kernels.launches - was, driver.kernel_counts()["generic"] - generic
        names = [e.name for e in prof.events() if "attention" in e.name]
        return said[1], len(names)

    assert counted([StepEntry("a", list(range(24)), [23])]) == (6, 6)
    entries = [StepEntry(i, [i + 1], [0]) for i in range(17)]
    assert counted(entries) == (3, 3)


@gpu
@pytest.mark.parametrize("activation,weight_on,identity,shared", [
    ("silu", "output", 0, False), ("silu", "output", 2, True), ("clamped_swish", "input", 0, False),
    ("clamped_swish", "output", 0, True), ("relu_squared", "output", 0, False)])
@pytest.mark.parametrize("rows,E,top,width,ff", [(520, 8, 2, 264, 272), (700, 5, 1, 128, 80), (1501, 4, 3, 64, 144)])
def test_routed_experts_of_many_rows(rows, E, top, width, ff, activation, weight_on, identity, shared):
    """The whole feed-forward with enough tokens per expert for the products on CTA pairs: the bits of
    the one-CTA products (one expert nearly without tokens, one with many), and the formula in float64."""
    from llmario_b200 import kernels
    from llmario_b200.config.spec import PartSpec
    from llmario_b200.parts.base import Segment, StepContext, Workspace, build_part
    assert kernels.moe_pairs(rows * top, E)
    b16 = lambda *s, seed: rnd(*s, dtype=torch.bfloat16, scale=s[-1] ** -0.5, seed=seed)  # noqa: E731
    gated = activation != "relu_squared"
    w = {"r": rnd(E + identity, width, scale=2 * width ** -0.5, seed=1)}
    names = {"router": ["r"]}
    for e in range(E):
        for k, shape in ((("gate", (ff, width)),) if gated else ()) + (("up", (ff, width)), ("down", (width, ff))):
            w[f"{k}{e}"] = b16(*shape, seed=10 * e + len(k))
            names[f"{k}{e}"] = [f"{k}{e}"]
    bias = torch.zeros(E + identity, device=DEV)
    bias[0], bias[1] = -3.0, 2.0
    w["b"], names["router_bias"] = bias, ["b"]
    params = dict(hidden_size=width, intermediate_size=ff, experts=E, top=top, identity=identity, activation=activation,
                  weight_on=weight_on, limit=0.7, scores="softmax_all" if identity else "softmax_chosen", tensors=names)
    if shared:
        for k, shape in (("gate", (32, width)), ("up", (32, width)), ("down", (width, 32))):
            w["s" + k] = b16(*shape, seed=99 + len(k))
        params["shared"] = PartSpec("swiglu", dict(hidden_size=width, intermediate_size=32,
                                                   tensors={k: ["s" + k] for k in ("gate", "up", "down")}))
    part = build_part("feed_forward", PartSpec("moe", params), w, torch.bfloat16, DEV)
    h = rnd(rows, width, dtype=torch.bfloat16, seed=3)
    x0 = rnd(rows, width, seed=4)
    ints = torch.zeros(rows, dtype=torch.int32, device=DEV)

    def forward():
        ctx = StepContext(rows=rows, tokens=ints, row_pos=ints, row_slot=ints, segments=[Segment("r", 0, 0, rows, 0)],
                          dtype=torch.bfloat16, device=torch.device(DEV), workspace=Workspace(torch.device(DEV)),
                          cache=None)
        x = x0.clone()
        part.forward(ctx, h, x)
        return x, ctx.buffer("moe.ids", (rows, top), torch.int32).clone(), \
            ctx.buffer("moe.weights", (rows, top), torch.float32).clone()

    got, ids, wts = forward()
    kernels.use_cta_pairs(False)
    try:
        lone, _, _ = forward()
    finally:
        kernels.use_cta_pairs(True)
    assert torch.equal(got, lone)
    kernels.check_tc_status(torch.device(DEV))
    hd, want = h.double(), x0.double()
    r16 = lambda t: t.to(torch.bfloat16).double()  # noqa: E731

    def act(z, e, s=1.0):
        up = z @ w[f"up{e}"].double().T * s
        if not gated:
            return r16(up.clamp(min=0) ** 2)
        g = z @ w[f"gate{e}"].double().T * s
        if activation == "silu":
            return r16(g * torch.sigmoid(g) * up)
        g, up = g.clamp(max=0.7), up.clamp(-0.7, 0.7)
        return r16(g * torch.sigmoid(1.702 * g) * (up + 1))

    for k in range(top):
        for e in range(E + identity):
            at = (ids[:, k] == e).nonzero()[:, 0]
            f = wts[at, k].double()[:, None]
            if e >= E:
                want[at] += f * hd[at]
            elif weight_on == "input":
                want[at] += act(hd[at], e, f) @ w[f"down{e}"].double().T
            else:
                want[at] += f * (act(hd[at], e) @ w[f"down{e}"].double().T)
    if shared:
        g = hd @ w["sgate"].double().T
        want += r16(g * torch.sigmoid(g) * (hd @ w["sup"].double().T)) @ w["sdown"].double().T
    # activations are rounded to 8 bits of mantissa on both sides: a rounding may fall the other way
    assert float((got.double() - want).norm() / (want - x0.double()).norm()) < 2 ** -9
