"""The kernels of the state mixers and of the window attention with pooled blocks, each alone against the plain
implementation's function for the same mechanism, on packed batches of unequal sequences, over several steps (the
state, the previous rows and the pooled rows come from the step before), on slots and pages in no particular order,
at sizes that fill a lane's registers unevenly.  Inputs are made so that one far key decides the result: a key that
is seen, not seen, or seen through its block changes the output by much more than any tolerance."""
import numpy as np
import pytest
import torch

import plain_sagizen as plain
from edgelm_b200.csrc import ops

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def i32(a):
    return torch.tensor(np.asarray(a), dtype=torch.int32, device=DEV)


def f32(a):
    return torch.tensor(np.asarray(a), dtype=torch.float32, device=DEV).contiguous()


def packed(lengths):
    tok0 = np.concatenate([[0], np.cumsum(lengths)])
    tok_seq = np.repeat(np.arange(len(lengths)), lengths)
    return i32(tok0), i32(tok_seq)


def steps_of(total, cuts):
    """Per step the (start, count) of every sequence: sequence s of length total[s] is fed in pieces of cuts[s]."""
    n_steps = max(len(c) for c in cuts)
    at = [0] * len(total)
    out = []
    for k in range(n_steps):
        step = []
        for s, c in enumerate(cuts):
            n = c[k] if k < len(c) else 0
            step.append((at[s], n))
            at[s] += n
        out.append(step)
    assert at == list(total)
    return out


@pytest.mark.parametrize("N,P,H,G", [(40, 12, 3, 3), (16, 8, 4, 2), (70, 5, 2, 1), (200, 3, 1, 1)])
def test_state_space_scan_over_steps(N, P, H, G):
    g = np.random.default_rng(N)
    total, cuts, slots = [43, 6, 1], [[5, 1, 37], [2, 4], [1]], [4, 0, 2]
    inner, C = H * P, H * P + 2 * G * N
    xbc = [g.normal(size=(n, C)) for n in total]
    dtr = [g.normal(size=(n, H)) for n in total]
    dt_bias, A_log, D = g.uniform(-1, 0.5, H), g.uniform(-4, -1, H), g.normal(size=H)
    want = [plain.ssm_recurrence(x[:, :inner].reshape(-1, H, P), x[:, inner:inner + G * N].reshape(-1, G, N), x[:, inner + G * N:].reshape(-1, G, N),
                                 plain.softplus(d + dt_bias), A_log, D, G).reshape(-1, inner) for x, d in zip(xbc, dtr)]
    state = torch.zeros(6, H, P, N, device=DEV)
    state[1].fill_(float("nan"))      # a slot of nobody: never read
    got = [np.zeros_like(w) for w in want]
    for step in steps_of(total, cuts):
        live = [(s, a, n) for s, (a, n) in enumerate(step) if n]
        tok0, _ = packed([n for _, _, n in live])
        x = f32(np.concatenate([xbc[s][a:a + n] for s, a, n in live]))
        u = f32(np.concatenate([dtr[s][a:a + n] for s, a, n in live]))
        y = torch.full((x.shape[0], inner), float("nan"), device=DEV)
        ops.ssm_scan(x, u, 0, f32(dt_bias), f32(A_log), f32(D), state, y, tok0, i32([slots[s] for s, _, _ in live]), len(live), H, G, N, P)
        y = y.cpu().numpy()
        at = 0
        for s, a, n in live:
            got[s][a:a + n] = y[at:at + n]
            at += n
    for w, o in zip(want, got):
        assert np.abs(o - w).max() < 2e-5 * max(1.0, np.abs(w).max())


@pytest.mark.parametrize("K,H", [(40, 2), (16, 3), (70, 1), (130, 1)])
def test_decayed_outer_product_scan_over_steps(K, H):
    g = np.random.default_rng(K)
    total, cuts, slots = [50, 3, 9], [[1, 2, 47], [3], [4, 4, 1]], [1, 3, 0]
    r, k, v = [[g.normal(size=(n, H, K)) * 0.5 for n in total] for _ in range(3)]
    w = [g.uniform(0.8, 0.999, size=(n, H, K)) for n in total]
    u = g.uniform(0, 1, size=(H, K))
    want = [plain.wkv_recurrence(r[s], k[s], v[s], w[s], u).reshape(-1, H * K) for s in range(3)]
    state = torch.zeros(5, H, K, K, device=DEV)
    got = [np.zeros_like(x) for x in want]
    for step in steps_of(total, cuts):
        live = [(s, a, n) for s, (a, n) in enumerate(step) if n]
        tok0, _ = packed([n for _, _, n in live])
        cat = lambda src: f32(np.concatenate([src[s][a:a + n].reshape(n, H * K) for s, a, n in live]))
        o = torch.full((int(tok0[-1]), H * K), float("nan"), device=DEV)
        ops.wkv_scan(cat(r), cat(k), cat(v), cat(w), f32(u), state, o, tok0, i32([slots[s] for s, _, _ in live]), len(live), H, K)
        o = o.cpu().numpy()
        at = 0
        for s, a, n in live:
            got[s][a:a + n] = o[at:at + n]
            at += n
    for x, o in zip(want, got):
        assert np.abs(o - x).max() < 2e-5 * max(1.0, np.abs(x).max())


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_blend_convolution_and_norms(dtype):
    g = np.random.default_rng(5)
    lengths, slots, D = [4, 1, 2], [2, 0, 1], 24
    tok0, tok_seq = packed(lengths)
    seqslot = i32(slots)
    x = g.normal(size=(7, D))
    prev = g.normal(size=(3, D))          # the state rows: what the step before left
    mu = g.uniform(0, 1, size=(5, D))
    state = f32(prev)
    out = torch.empty(5, 7, D, dtype=dtype, device=DEV)
    xin = f32(x).to(dtype)
    ops.shift_mix(xin, state, f32(mu), out, tok_seq, tok0, seqslot)
    xr = xin.float().cpu().numpy().astype(np.float64)
    before = np.concatenate([np.concatenate([prev[slots[s]][None].astype(np.float32), xr[a:b - 1]]) for s, (a, b) in enumerate(zip(tok0.tolist(), tok0.tolist()[1:]))])
    want = xr[None] + (before - xr)[None] * mu[:, None].astype(np.float32)
    tol = 1e-6 if dtype == torch.float32 else 2e-2
    assert np.abs(out.float().cpu().numpy() - want).max() < tol
    ops.save_last_rows(xin, state, tok0, seqslot, 3)
    assert np.array_equal(state.cpu().numpy()[slots], xr[[3, 4, 6]].astype(np.float32))
    # convolution: taps 4, steps of 4, 1 and 2 tokens on top of a tail of 3 rows
    C, taps = 10, 4
    u = g.normal(size=(7, C + 3))
    w, b = g.normal(size=(C, taps)), g.normal(size=C)
    tail = g.normal(size=(3, taps - 1, C))
    cstate = f32(tail)
    y = torch.empty(7, C, device=DEV)
    ops.conv_silu(f32(u), 2, f32(w), f32(b), cstate, y, tok_seq, tok0, seqslot, 3)
    for s, (a, e) in enumerate(zip(tok0.tolist(), tok0.tolist()[1:])):
        full = np.concatenate([tail[slots[s]], u[a:e, 2:2 + C]])
        ref = plain.causal_conv_silu(full, w, b)[taps - 1:]
        assert np.abs(y[a:e].cpu().numpy() - ref).max() < 1e-5
        assert np.allclose(cstate[slots[s]].cpu().numpy(), full[-(taps - 1):], atol=1e-6)
    # gated group norm, both orders; the norm on a sublayer's output with the residual sum
    yv, gate, wn = g.normal(size=(7, 24)), g.normal(size=(7, 30)), g.uniform(0.5, 1.5, 24)
    for first in (True, False):
        o = torch.empty(7, 24, dtype=dtype, device=DEV)
        ops.gated_group_norm(f32(yv), f32(gate)[:, 3:27], f32(wn), o, 3, 1e-4, first)
        gt = plain.silu(gate[:, 3:27])
        ref = plain.unit_rms((yv * gt).reshape(7, 3, 8), 1e-4).reshape(7, 24) * wn if first else plain.unit_rms(yv.reshape(7, 3, 8), 1e-4).reshape(7, 24) * wn * gt
        assert np.abs(o.float().cpu().numpy() - ref).max() < (1e-5 if dtype == torch.float32 else 3e-2)
    xs, y1, y2 = g.normal(size=(7, 24)), g.normal(size=(7, 24)), g.normal(size=(7, 24))
    xd, cast = f32(xs), torch.empty(7, 24, dtype=dtype, device=DEV)
    ops.rmsnorm_add(xd, f32(y1), f32(wn), 1e-3, a=1.2, y2=f32(y2), b=0.7, cast=cast)
    ref = xs + plain.rmsnorm(1.2 * y1 + 0.7 * y2, wn, 1e-3)
    assert np.abs(xd.cpu().numpy() - ref).max() < 1e-5 and np.abs(cast.float().cpu().numpy() - ref).max() < (1e-5 if dtype == torch.float32 else 3e-2)
    a = g.normal(size=(7, 6))
    w2, w0 = g.normal(size=(24, 6)), g.uniform(-4, -1, 24)
    dec = torch.empty(7, 24, device=DEV)
    w2d = f32(w2).to(dtype)
    ops.lowrank_decay(f32(a), w2d, f32(w0), dec)
    ref = np.exp(-np.exp(np.tanh(a) @ w2d.float().cpu().numpy().astype(np.float64).T + w0))
    assert np.abs(dec.cpu().numpy() - ref).max() < 1e-5


@pytest.mark.parametrize("C,taps,bias,act", [(260, 4, True, "silu"), (64, 2, False, None), (512, 1, True, "silu"), (1028, 3, True, None),
                                             (18948, 4, True, "silu"), (18948, 3, False, None), (19200, 2, True, None), (18948, 1, True, "silu")])
def test_filter_over_many_tokens(C, taps, bias, act):
    """Steps of more than 64 tokens, few channels and enough for the kernel of many tokens: sequences that start inside a run of tokens,
    shorter than the filter, going on from a tail."""
    g = np.random.default_rng(C)
    lengths, slots = [70, 1, 2, 33], [3, 0, 5, 2]
    u, w, b, ib, tail = g.normal(size=(106, C + 8)), g.normal(size=(C, taps)), g.normal(size=C), g.normal(size=C), g.normal(size=(6, taps - 1, C))
    tok0, tok_seq = packed(lengths)
    state, y = f32(tail), torch.full((106, C), float("nan"), device=DEV)
    ops.conv_act(f32(u), 4, f32(w), f32(b) if bias else None, state, y, tok_seq, tok0, i32(slots), 4, in_bias=f32(ib), act=act)
    for s, (a, e) in enumerate(zip(tok0.tolist(), tok0.tolist()[1:])):
        full = np.concatenate([tail[slots[s]], u[a:e, 4:4 + C] + ib])
        ref = sum(full[j:j + e - a] * w[:, j] for j in range(taps)) + (b if bias else 0.0)
        ref = plain.silu(ref) if act else ref
        assert np.abs(y[a:e].cpu().numpy() - ref).max() < 3e-6 * max(1.0, np.abs(ref).max())      # (five roundings of sums up to 16)
        if taps > 1:
            assert np.allclose(state[slots[s]].cpu().numpy(), full[-(taps - 1):], atol=1e-6)


@pytest.mark.parametrize("taps", [1, 2, 3, 4])
@pytest.mark.parametrize("cut", [0, 21, 23])
def test_filter_reads_no_token_in_front_of_its_taps(taps, cut):
    """An infinity and a NaN reach `taps` tokens each, in one step and where the step is cut behind the infinity."""
    g = np.random.default_rng(taps)
    T, C, bad = 180, 13400, {20: np.inf, 99: np.nan}        # (channels enough for the kernel of many tokens)
    u, w = g.normal(size=(T, C)), g.normal(size=(C, taps)) + 2.0
    for t, value in bad.items():
        u[t, 5] = value
    state, got = torch.zeros(1, taps - 1, C, device=DEV), []
    for a, e in ((0, cut), (cut, T)):
        if a == e:
            continue
        tok0, tok_seq = packed([e - a])
        y = torch.empty(e - a, C, device=DEV)
        ops.conv_act(f32(u[a:e]), 0, f32(w), None, state, y, tok_seq, tok0, i32([0]), 1)
        got.append(y.isfinite().cpu().numpy())
    want = np.ones((T, C), bool)
    for t in bad:
        want[t:t + taps, 5] = False
    assert (np.concatenate(got) == want).all()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("gs,groups", [(4, 3), (64, 5), (128, 2), (100, 3), (576, 1), (1028, 2), (4096, 1), (8192, 1), (8200, 1), (66, 2)])
def test_gated_group_norm_of_many_rows(gs, groups, dtype):
    """Every way a group is shared by threads, the last one ragged; sizes that no vector form takes too."""
    g = np.random.default_rng(gs)
    T, inner = 67, gs * groups
    y, gate, w = g.normal(size=(T, inner)), g.normal(size=(T, inner + 4)), g.uniform(0.5, 1.5, inner)
    for first in (True, False):
        for act in ("silu", "sigmoid"):
            o = torch.full((T, inner), float("nan"), dtype=dtype, device=DEV)
            ops.gated_group_norm(f32(y), f32(gate)[:, 4:], f32(w), o, groups, 1e-4, first, gate_act=act)
            a = plain.silu(gate[:, 4:]) if act == "silu" else 1.0 / (1.0 + np.exp(-gate[:, 4:]))
            norm = lambda v: plain.unit_rms(v.reshape(T, groups, gs), 1e-4).reshape(T, inner) * w
            ref = norm(y * a) if first else norm(y) * a
            off = np.abs(o.float().cpu().numpy() - ref)
            assert (off < 3e-6 * max(1.0, np.abs(ref).max()) + (0 if dtype == torch.float32 else 2.0 ** -8 * np.abs(ref))).all()


def chunk_steps(total, cuts):
    """Per step the sequences' new tokens, `seq_tok0` and the tiles of STATE_CHUNK tokens (first row, tokens, count)."""
    from edgelm_b200.engine.batch import make_tiles
    for step in steps_of(total, cuts):
        n_new = [n for _, n in step]
        _, tok0, ntok, _ = make_tiles(n_new, [0] * len(n_new), ops.STATE_CHUNK)
        yield step, packed(n_new)[0], (i32(tok0), i32(ntok), len(tok0))


def rows_of(xs, step):
    return np.concatenate([x[a:a + n].reshape(n, int(np.prod(x.shape[1:]))) for x, (a, n) in zip(xs, step)])


CHUNK_TOTAL, CHUNK_CUTS = [200, 64, 65, 131], [[129, 71], [64], [1, 64], [0, 128, 3]]


@pytest.mark.parametrize("H,G,N,P", [(4, 1, 128, 64), (4, 2, 16, 20), (3, 3, 60, 64), (2, 1, 100, 4)])
def test_state_space_chunk_by_chunk(H, G, N, P):
    """Edges of chunks, sequences without a token in a step, states from earlier pieces, decays from nearly 1 to zero; 2^-24 of the largest
    value for each term of the three sums behind an output (64 tokens, N state rows, 64 again), and twice that in the state."""
    g = np.random.default_rng(N + P)
    total = CHUNK_TOTAL
    x, B, C = [g.normal(size=(n, H, P)) for n in total], [g.normal(size=(n, G, N)) for n in total], [g.normal(size=(n, G, N)) / np.sqrt(N) for n in total]
    raw = [g.normal(-3, 2, size=(n, H)) for n in total]
    raw[0][77] = 200.0
    bias, A_log, D = g.normal(size=H), g.uniform(-2, 2, H), g.normal(size=H)
    want = [plain.ssm_recurrence(a, b, c, plain.softplus(r + bias), A_log, D, G) for a, b, c, r in zip(x, B, C, raw)]
    slots, states = [3, 0, 5, 2], [torch.zeros(6, H, P, N, device=DEV) for _ in range(2)]
    for s in states:
        s[1] = s[4] = 7.0                       # (slots of nobody)
    worst, squares, scale = [0.0, 0.0], [0.0, 0.0], max(np.abs(w).max() for w in want)
    for step, tok0, tiles in chunk_steps(total, CHUNK_CUTS):
        xbc, u = f32(np.concatenate([rows_of(x, step), rows_of(B, step), rows_of(C, step)], 1)), f32(np.pad(rows_of(raw, step), ((0, 0), (3, 2))))
        for i, s in enumerate(states):
            y = torch.full((len(xbc), H * P), float("nan"), device=DEV)
            args = (xbc, u, 3, f32(bias), f32(A_log), f32(D), s, y, tok0, i32(slots), 4)
            if i == 0:
                ops.ssm_chunked(*args, *tiles, H, G, N, P)
            else:
                ops.ssm_scan(*args, H, G, N, P)
            off = y.cpu().numpy() - rows_of(want, step)
            worst[i], squares[i] = max(worst[i], np.abs(off).max()), squares[i] + (off ** 2).sum()
    assert squares[0] <= 1.1 * squares[1], squares     # (no further from float64 than the walk; the few largest values make the sums: 5 % of a root are chance)
    assert worst[0] < (128 + N) * 2.0 ** -24 * scale, worst
    assert float((states[0] - states[1]).abs().max()) < 2 * (128 + N) * 2.0 ** -24 * max(1.0, float(states[1][slots].abs().max()))
    assert bool((states[0][1] == 7).all() and (states[0][4] == 7).all())


NOT_FINITE = {"rate": ("A_log", (1,), 100.0), "rate_nan": ("A_log", (1,), np.nan), "bias_nan": ("dt_bias", (2,), np.nan), "step": ("raw", (58, 1), np.inf),
              "step_nan": ("raw", (57, 1), np.nan), "x": ("x", (57, 1, 3), np.inf), "x_nan": ("x", (30, 0, 7), np.nan), "B": ("B", (57, 0, 2), -np.inf),
              "C": ("C", (57, 0, 2), np.nan)}


@pytest.mark.parametrize("what", NOT_FINITE)
def test_state_space_chunks_are_finite_where_the_walk_is(what):
    """... and agree with it there (2e-5: the bound of the walk beside float64)."""
    from edgelm_b200.engine.batch import make_tiles
    g = np.random.default_rng(3)
    lengths, H, G, N, P = [20, 150], 3, 1, 16, 8
    T = sum(lengths)
    c = {"x": g.normal(size=(T, H, P)), "B": g.normal(size=(T, G, N)), "C": g.normal(size=(T, G, N)), "raw": g.normal(-3, 1, size=(T, H)),
         "A_log": g.uniform(-1, 1, H), "dt_bias": g.normal(size=H)}
    name, at, value = NOT_FINITE[what]
    c[name][at] = value
    xbc, tok0 = f32(np.concatenate([c[k].reshape(T, -1) for k in ("x", "B", "C")], 1)), packed(lengths)[0]
    _, ttok0, tntok, _ = make_tiles(lengths, [0, 0], ops.STATE_CHUNK)
    outs = []
    for chunked in (True, False):
        state, y = torch.zeros(2, H, P, N, device=DEV), torch.full((T, H * P), float("nan"), device=DEV)
        args = (xbc, f32(c["raw"]), 0, f32(c["dt_bias"]), f32(c["A_log"]), f32(np.ones(H)), state, y, tok0, i32([1, 0]), 2)
        if chunked:
            ops.ssm_chunked(*args, i32(ttok0), i32(tntok), len(ttok0), H, G, N, P)
        else:
            ops.ssm_scan(*args, H, G, N, P)
        outs.append((y.isfinite(), state.isfinite(), y.nan_to_num(0, 0, 0)))
    assert torch.equal(outs[0][0], outs[1][0]) and torch.equal(outs[0][1], outs[1][1])
    assert float((outs[0][2] - outs[1][2]).abs().max()) < 2e-5 * float(outs[1][2].abs().max())


@pytest.mark.parametrize("H,K", [(3, 64), (2, 20), (1, 4), (2, 36)])
def test_time_mix_chunk_by_chunk(H, K):
    """As above for a decay per key channel, down to zero: 64 terms of the walk, K of the product, in each output."""
    g = np.random.default_rng(K)
    total = CHUNK_TOTAL
    r, k, v = ([g.normal(size=(n, H, K)) for n in total] for _ in range(3))
    w = [np.float32(np.exp(-np.exp(g.uniform(-8, 2, size=(n, H, K))))).astype(np.float64) for n in total]
    w[0][77] = 0.0
    bonus = g.normal(size=(H, K))
    want = [plain.wkv_recurrence(a, b, c, d, bonus) for a, b, c, d in zip(r, k, v, w)]
    slots, states = [3, 0, 5, 2], [torch.zeros(6, H, K, K, device=DEV) for _ in range(2)]
    for s in states:
        s[1] = s[4] = 7.0                       # (slots of nobody)
    worst, squares, scale = [0.0, 0.0], [0.0, 0.0], max(np.abs(x).max() for x in want)
    for step, tok0, tiles in chunk_steps(total, CHUNK_CUTS):
        rows = [f32(rows_of(x, step)) for x in (r, k, v, w)]
        for i, s in enumerate(states):
            o = torch.full_like(rows[0], float("nan"))
            if i == 0:
                ops.wkv_chunked(*rows, f32(bonus), s, o, tok0, i32(slots), 4, *tiles, H, K)
            else:
                ops.wkv_scan(*rows, f32(bonus), s, o, tok0, i32(slots), 4, H, K)
            off = o.cpu().numpy() - rows_of(want, step)
            worst[i], squares[i] = max(worst[i], np.abs(off).max()), squares[i] + (off ** 2).sum()
    assert squares[0] <= 1.1 * squares[1], squares     # (no further from float64 than the walk; the few largest values make the sums: 5 % of a root are chance)
    assert worst[0] < (64 + K) * 2.0 ** -24 * scale, worst
    assert float((states[0] - states[1]).abs().max()) < (64 + K) * 2.0 ** -24 * max(1.0, float(states[1][slots].abs().max()))
    assert bool((states[0][1] == 7).all() and (states[0][4] == 7).all())


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("T,C,L", [(1, 130, 5), (37, 2048, 64), (333, 1000, 24), (160, 2048, 513), (2500, 128, 7)])
def test_lowrank_decay_tiles(T, C, L, dtype):
    """One and sixteen tokens a block, ragged edges of both, ranks in and out of whole pieces.  The sum takes L
    roundings of 2^-24 of partial sums under 2, of which exp(-exp(.)) passes on at most 0.37, and its own functions eight more."""
    g = np.random.default_rng(T + L)
    a, w2, w0 = g.normal(size=(T, L)), f32(g.normal(size=(C, L)) / np.sqrt(L)).to(dtype), g.uniform(-4, 1, C)
    out = torch.full((T, C), float("nan"), device=DEV)
    ops.lowrank_decay(f32(a), w2, f32(w0), out)
    ref = torch.exp(-torch.exp(torch.tanh(f32(a).double()) @ w2.double().T + f32(w0).double()))
    assert float((out.double() - ref).abs().max()) < (L + 8) * 2.0 ** -24


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("window,pool,dk,dv,H,G", [(9, 4, 20, 12, 4, 2), (3, 7, 40, 72, 2, 1), (70, 64, 16, 16, 3, 3), (5, 1, 33, 8, 2, 2)])
def test_window_attention_with_pooled_blocks(dtype, window, pool, dk, dv, H, G):
    """Two sequences side by side through prompt pieces and single tokens.  In the first, key 37 (its block too) is far
    larger than every other along the direction all queries point in: where it is seen it takes almost all the weight."""
    g = np.random.default_rng(window * 100 + pool)
    PAGE = 64
    total = [150, 70]
    cuts = [[41] + [1] * 19 + [90], [1, 2, 3] + [1] * 17 + [47]]
    q = [g.normal(size=(n, H, dk)) * 0.3 for n in total]
    k = [g.normal(size=(n, G, dk)) * 0.3 for n in total]
    v = [g.normal(size=(n, G, dv)) for n in total]
    q[0][:, :, 0] += 3.0
    k[0][37, :, 0] += 12.0
    scale = 0.5
    rnd = lambda a: f32(a).to(dtype).float().cpu().numpy().astype(np.float64)     # what the cache holds
    want = [plain.pooled_window_attention(rnd(q[s]), rnd(k[s]), rnd(v[s]), scale, window, pool).reshape(total[s], H * dv) for s in range(2)]
    w0 = want[0].reshape(150, H, dv)
    seen_as_token, unseen, seen_as_block = 37 + window - 1, 37 + window, (37 // pool) * pool + pool - 1 + window
    if seen_as_block > unseen:     # (the block is complete and behind the window later than the token leaves it)
        assert np.abs(w0[seen_as_token] - w0[unseen]).max() > 0.3 and np.abs(w0[seen_as_block] - w0[seen_as_block - 1]).max() > 0.05
    n_pages, R = 8, -(-PAGE // pool)
    kc = torch.full((n_pages, G, PAGE, dk), float("nan"), dtype=dtype, device=DEV)
    vc = torch.full((n_pages, G, PAGE, dv), float("nan"), dtype=dtype, device=DEV)
    pk = torch.full((n_pages, G, R, dk), float("nan"), device=DEV)
    pv = torch.full((n_pages, G, R, dv), float("nan"), device=DEV)
    table = i32([[5, 2, 7, -1], [0, 6, -1, -1]])
    err = torch.zeros(1, dtype=torch.int32, device=DEV)
    got = [np.zeros_like(w) for w in want]
    got_tiled = [np.zeros_like(w) for w in want]
    for step in steps_of(total, cuts):
        live = [(s, a, n) for s, (a, n) in enumerate(step) if n]
        T = sum(n for _, _, n in live)
        tok_pos = i32(np.concatenate([np.arange(a, a + n) for _, a, n in live]))
        tok_seq = i32(np.concatenate([np.full(n, s) for s, _, n in live]))     # rows of the page table: here the sequences themselves
        qkv = f32(np.concatenate([np.concatenate([q[s][a:a + n].reshape(n, -1), k[s][a:a + n].reshape(n, -1), v[s][a:a + n].reshape(n, -1)], 1) for s, a, n in live]))
        qd = torch.empty(T, H * dk, dtype=dtype, device=DEV)
        ops.qk_rope_norm_append(qkv, None, qd, tok_pos, tok_seq, table, kc, vc, H, G, dk, dv, 0, None, 0.0, False, err)
        ops.pool_blocks(tok_pos, tok_seq, table, kc, vc, pk, pv, T, G, dk, dv, pool, err)
        out = torch.full((T, H * dv), float("nan"), dtype=dtype, device=DEV)
        ops.pooled_window_attn(qd, out, kc, vc, pk, pv, tok_pos, tok_seq, table, H, G, dk, dv, scale, window, pool)
        # the prompt kernel on the same step: runs of at most 32 / (H / G) tokens, 32 rows a block
        from edgelm_b200.engine.batch import make_tiles
        tile_tokens = max(1, 32 // (H // G))
        assert [s for s, _, _ in live] == list(range(len(live)))      # (a tile's sequence index is its row of the page table)
        cols = make_tiles([n for _, _, n in live], [a for _, a, _ in live], tile_tokens)
        out_t = torch.full((T, H * dv), float("nan"), dtype=dtype, device=DEV)
        ops.pooled_window_attn_tiled(qd, out_t, kc, vc, pk, pv, table, i32(cols[0]), i32(cols[1]), i32(cols[2]), i32(cols[3]), len(cols[0]),
                                     tile_tokens, H, G, dk, dv, scale, window, pool)
        out, out_t = out.float().cpu().numpy(), out_t.float().cpu().numpy()
        at = 0
        for s, a, n in live:
            got[s][a:a + n] = out[at:at + n]
            got_tiled[s][a:a + n] = out_t[at:at + n]
            at += n
    assert int(err.item()) == 0
    tol = 2e-5 if dtype == torch.float32 else 2e-2
    for w, o, ot in zip(want, got, got_tiled):
        assert np.isfinite(o).all() and np.abs(o - w).max() < tol * max(1.0, np.abs(w).max())
        assert np.isfinite(ot).all() and np.abs(ot - w).max() < tol * max(1.0, np.abs(w).max())


@pytest.mark.parametrize("window,pool,d,H,G", [(9, 4, 64, 4, 2), (70, 64, 32, 3, 3), (33, 1, 128, 2, 1), (64, 5, 64, 3, 1), (40, 7, 128, 2, 2)])
def test_window_attention_of_whole_rows(window, pool, d, H, G):
    """Heads that the kernel of whole rows takes: runs of keys and of pooled rows that are empty, a part of a load and several loads."""
    for dtype in (torch.float32, torch.bfloat16):
        test_window_attention_with_pooled_blocks(dtype, window, pool, d, d, H, G)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("window,pool,d", [(9, 4, 20), (40, 7, 96), (1, 4, 64), (40, 7, 32), (33, 1, 64), (70, 64, 128), (300, 5, 64)])
def test_window_attention_of_single_tokens_that_see_no_number(window, pool, d, dtype):
    """One sequence a fault: a not-a-number or an infinity in a key, a value or a pooled row that the token sees, in its query, or (the last ones) where
    it does not see it.  What the token's heads are then is what 64 bits give (not-a-numbers at the same places, infinities with their sign),
    also where the faulty score is the only one of a warp's run (window 1: of the whole window).  Scores stay under 30, so no weight is zero."""
    g = np.random.default_rng(window + d)
    PAGE, n, H, G = 64, 150, 4, 2
    R, pages = -(-PAGE // pool), -(-n // PAGE)
    seen_blocks = max(0, (n - window) // pool)
    bad = [("k", n - 1, np.nan), ("k", max(0, n - window), np.nan), ("k", n - 1, np.inf), ("k", n - 1, -np.inf), ("v", n - 1, np.nan), ("v", n - 1, -np.inf),
           ("q", 0, np.nan), ("none", 0, 0.0)]
    if seen_blocks:
        bad += [("pk", 0, np.nan), ("pk", seen_blocks - 1, -np.inf), ("pv", seen_blocks // 2, np.inf), ("pv", 0, np.nan), ("k", n - window - 1, np.nan)]
    B, scale = len(bad), d ** -0.5
    q, kc, vc = g.normal(size=(B, H, d)), np.full((B * pages, G, PAGE, d), np.nan), np.full((B * pages, G, PAGE, d), np.nan)
    pk, pv = np.full((B * pages, G, R, d), np.nan), np.full((B * pages, G, R, d), np.nan)
    rnd = lambda a: torch.tensor(a).to(dtype).double().numpy()
    want = np.zeros((B, H, d))
    for s, (what, at, value) in enumerate(bad):
        k, v, bk, bv = (g.normal(size=(m, G, d)) for m in (n, n, n // pool, n // pool))
        {"k": k, "v": v, "pk": bk, "pv": bv, "q": q[s][None], "none": k}[what][at, :, 3] += value
        for i in range(n):
            kc[s * pages + i // PAGE, :, i % PAGE], vc[s * pages + i // PAGE, :, i % PAGE] = k[i], v[i]
        for e in range(n // pool):
            end = (e * pool + pool - 1) // PAGE
            pk[s * pages + end, :, e - PAGE * end // pool], pv[s * pages + end, :, e - PAGE * end // pool] = bk[e], bv[e]
        lo = max(0, n - window)
        keys = np.concatenate([rnd(k[lo:]), np.float32(bk[:seen_blocks]).astype(np.float64)])
        vals = np.concatenate([rnd(v[lo:]), np.float32(bv[:seen_blocks]).astype(np.float64)])
        for h in range(H):
            sc = torch.tensor(keys[:, h // 2]) @ torch.tensor(rnd(q[s, h])) * scale
            want[s, h] = (torch.softmax(sc, 0)[:, None] * torch.tensor(vals[:, h // 2])).sum(0).numpy()
    out = torch.full((B, H * d), 7.0, dtype=dtype, device=DEV)
    cast = lambda a: f32(a).to(dtype)
    ops.pooled_window_attn(cast(q.reshape(B, -1)), out, cast(kc), cast(vc), f32(pk), f32(pv), i32([n - 1] * B), i32(list(range(B))),
                           i32([[s * pages + i for i in range(pages)] for s in range(B)]), H, G, d, d, scale, window, pool)
    got = out.float().cpu().numpy().reshape(B, H, d)
    assert np.isnan(want[:2]).all() and np.isnan(want[6]).all() and np.isfinite(want[7]).all() and (not seen_blocks or np.isfinite(want[-1]).all())
    for s, fault in enumerate(bad):
        assert np.array_equal(np.isnan(got[s]), np.isnan(want[s])) and np.array_equal(np.isinf(got[s]), np.isinf(want[s])), fault
        assert np.array_equal(got[s][np.isinf(got[s])], want[s][np.isinf(got[s])]), fault
        there = np.isfinite(want[s])
        assert np.abs(got[s][there] - want[s][there]).max(initial=0.0) < (2e-5 if dtype == torch.float32 else 2e-2) * 4, fault


@pytest.mark.parametrize("window,pool,d,H,G", [(100, 64, 64, 4, 2), (7, 3, 32, 3, 1), (64, 1, 96, 2, 2), (200, 5, 128, 2, 1), (50, None, 64, 2, 1)])
def test_pooled_attention_on_the_tensor_cores(window, pool, d, H, G):
    """Prompts and pieces that go on from the cache, up to 300 pooled rows, edges of pages and tiles, unwritten rows poisoned.  The
    output's bfloat16 rounding is 2^-9 of a value; beside the CUDA-core kernel, whose float32 sums differ in order only, a rounding
    may fall the other way where a sum lies within 2^-20 of its edge (a share of 2^-9, measured under 0.002)."""
    from edgelm_b200.engine.batch import make_tiles
    g = np.random.default_rng(window)
    PAGE, total, scale = 64, [333, 64, 1], 1.3 / np.sqrt(d)
    bf = lambda a: torch.tensor(a, dtype=torch.bfloat16).double().numpy()
    q = [bf(g.normal(size=(n, H, d)) * 2) for n in total]
    k, v = ([bf(g.normal(size=(n, G, d))) for n in total] for _ in range(2))
    want = [plain.pooled_window_attention(a, b, c, scale, window, pool) for a, b, c in zip(q, k, v)]
    R = -(-PAGE // pool) if pool else 1
    kc, vc = (torch.full((9, G, PAGE, d), float("nan"), dtype=torch.bfloat16, device=DEV) for _ in range(2))
    pk, pv = (torch.full((9, G, R, d), float("nan"), device=DEV) for _ in range(2))
    table, err = i32([[5, 2, 7, 8, 1, 3], [0] + [-1] * 5, [6] + [-1] * 5]), torch.zeros(1, dtype=torch.int32, device=DEV)
    assert ops.pooled_window_attn_mma_takes(torch.bfloat16, d, d)
    for step in steps_of(total, [[70, 1, 63, 199], [5, 2, 57], [1]]):
        live = [(s, a, n) for s, (a, n) in enumerate(step) if n]
        T = sum(n for _, _, n in live)
        pos, seq = i32(np.concatenate([np.arange(a, a + n) for _, a, n in live])), i32(np.concatenate([np.full(n, s) for s, _, n in live]))
        row = lambda s, a, n: np.concatenate([x[s][a:a + n].reshape(n, -1) for x in (q, k, v)], 1)
        qd = torch.empty(T, H * d, dtype=torch.bfloat16, device=DEV)
        ops.qk_rope_norm_append(f32(np.concatenate([row(*l) for l in live])), None, qd, pos, seq, table, kc, vc, H, G, d, d, 0, None, 0.0, False, err)
        if pool:
            ops.pool_blocks(pos, seq, table, kc, vc, pk, pv, T, G, d, d, pool, err)
        outs = []
        for tokens in (64, max(1, 32 // (H // G))):
            cols = make_tiles([n for _, _, n in live], [a for _, a, _ in live], tokens)
            out = torch.full((T, H * d), float("nan"), dtype=torch.bfloat16, device=DEV)
            call = (qd, out, kc, vc, pk if pool else None, pv if pool else None, table[[s for s, _, _ in live]].contiguous(), *map(i32, cols), len(cols[0]))
            if tokens == 64:
                ops.pooled_window_attn_mma(*call, H, G, d, d, scale, window, pool)
            else:
                ops.pooled_window_attn_tiled(*call, tokens, H, G, d, d, scale, window, pool)
            outs.append(out.float().cpu().numpy())
        ref = np.concatenate([want[s][a:a + n].reshape(n, -1) for s, a, n in live])
        assert np.abs(outs[0] - ref).max() < 2.0 ** -8 * np.abs(ref).max()
        assert (np.abs(outs[0] - ref) <= 2.0 ** -8 * np.abs(ref) + 1e-5).all()
        assert (outs[0] != outs[1]).mean() < 0.01
    assert int(err.item()) == 0


@pytest.mark.parametrize("pool,G", [(1, 1), (1, 20), (3, 16), (7, 2), (16, 1), (64, 2), (100, 3)])
def test_pooled_rows_of_many_tokens(pool, G):
    """Runs of one token to sixteen a block, with none, one and several ends of blocks in a run; sequences that start inside a run, one of
    them going on; a mean of 100 values in float32."""
    g = torch.Generator().manual_seed(pool)
    lengths, first, d = [170, 33, 97], [0, 5, 150], 20
    pos, seq = (np.concatenate(x) for x in ([np.arange(a, a + n) for a, n in zip(first, lengths)], [np.full(n, s) for s, n in enumerate(lengths)]))
    R = -(-64 // pool)
    kc, vc = (torch.randn(8, G, 64, d, generator=g).to(DEV) for _ in range(2))
    pk, pv = (torch.full((8, G, R, d), float("nan"), device=DEV) for _ in range(2))
    table, err = i32([[5, 2, 7, -1], [0, -1, -1, -1], [6, 1, 3, 4]]), torch.zeros(1, dtype=torch.int32, device=DEV)
    ops.pool_blocks(i32(pos), i32(seq), table, kc, vc, pk, pv, len(pos), G, d, d, pool, err)
    want = {}
    for p, s in zip(pos, seq):
        if (p + 1) % pool == 0:
            b, rows = p // pool, [(int(table[s, j // 64]), j % 64) for j in range(p + 1 - pool, p + 1)]
            want[(int(table[s, p // 64]), int(b - 64 * (p // 64) // pool))] = rows
    for got, c in ((pk, kc.cpu()), (pv, vc.cpu())):
        written = (~got.isnan()).all(-1).all(1).cpu()
        assert sorted(map(tuple, written.nonzero().tolist())) == sorted(want)
        for (page, row), rows in want.items():
            mean = torch.stack([c[a, :, j].double() for a, j in rows]).mean(0)
            assert float((got[page, :, row].cpu().double() - mean).abs().max()) < 1e-6
    assert int(err.item()) == 0


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_rotation_bias_and_unit_norm(dtype):
    g = np.random.default_rng(9)
    H, G, dk, dv, rot, eps = 3, 1, 20, 6, 12, 1e-4
    pos = np.array([0, 1, 63, 64, 1000, 250000])
    T = len(pos)
    qkv = g.normal(size=(T, (H + G) * dk + G * dv))
    bias = g.normal(size=qkv.shape[1])
    freq = 1e4 ** (-2.0 * np.arange(rot // 2) / rot) / 3.0
    n_pages = 250000 // 64 + 1
    kc = torch.zeros((n_pages, G, 64, dk), dtype=dtype, device=DEV)
    vc = torch.zeros((n_pages, G, 64, dv), dtype=dtype, device=DEV)
    table = torch.arange(n_pages, dtype=torch.int32, device=DEV).view(1, -1)
    qd = torch.empty(T, H * dk, dtype=dtype, device=DEV)
    err = torch.zeros(1, dtype=torch.int32, device=DEV)
    ops.qk_rope_norm_append(f32(qkv), f32(bias), qd, i32(pos), i32(np.zeros(T)), table, kc, vc, H, G, dk, dv, rot,
                            torch.tensor(freq, dtype=torch.float64, device=DEV), eps, True, err)
    x = qkv.astype(np.float32).astype(np.float64) + bias.astype(np.float32)
    qk = plain.unit_rms(plain.rotate_partial(x[:, :(H + G) * dk].reshape(T, H + G, dk), pos, rot, 1e4, 3.0), eps)
    tol = 3e-6 if dtype == torch.float32 else 2e-2
    assert np.abs(qd.float().cpu().numpy().reshape(T, H, dk) - qk[:, :H]).max() < tol
    for i, p in enumerate(pos):
        assert np.abs(kc[p // 64, 0, p % 64].float().cpu().numpy() - qk[i, H]).max() < tol
        assert np.abs(vc[p // 64, 0, p % 64].float().cpu().numpy() - x[i, (H + G) * dk:]).max() < tol
    assert int(err.item()) == 0


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("H,G,dk,dv,rot", [(66, 3, 64, 64, 64), (68, 2, 64, 64, 32), (68, 1, 128, 128, 64), (66, 2, 96, 192, 0)])
def test_rotation_bias_and_unit_norm_of_many_tokens(H, G, dk, dv, rot, dtype):
    """Heads of whole runs of 32 in steps of more than 64 tokens, two sequences, the last run of tokens a part.  3e-6: a dozen float32
    roundings of values up to 5 (a unit row's largest); a bfloat16 value is off by 2^-9 of itself beside that."""
    g = np.random.default_rng(dk + rot)
    eps, lengths, first = 1e-4, [70, 130], [0, 1000]
    T, pos = sum(lengths), np.concatenate([np.arange(a, a + n) for a, n in zip(first, lengths)])
    qkv, bias = g.normal(size=(T, (H + G) * dk + G * dv)), g.normal(size=(H + G) * dk + G * dv)
    freq = 1e4 ** (-2.0 * np.arange(rot // 2) / max(rot, 1)) / 3.0
    kc, vc = (torch.zeros((5, G, 64, d), dtype=dtype, device=DEV) for d in (dk, dv))
    table = torch.full((2, 18), -1, dtype=torch.int32, device=DEV)
    table[0, :2], table[1, 15:18] = i32([3, 0]), i32([4, 1, 2])
    seq = np.repeat([0, 1], lengths)
    qd, err = torch.full((T, H * dk), float("nan"), dtype=dtype, device=DEV), torch.zeros(1, dtype=torch.int32, device=DEV)
    ops.qk_rope_norm_append(f32(qkv), f32(bias), qd, i32(pos), i32(seq), table, kc, vc, H, G, dk, dv, rot,
                            torch.tensor(freq, dtype=torch.float64, device=DEV) if rot else None, eps, True, err)
    x = qkv.astype(np.float32).astype(np.float64) + bias.astype(np.float32)
    qk = x[:, :(H + G) * dk].reshape(T, H + G, dk)
    qk = plain.unit_rms(plain.rotate_partial(qk, pos, rot, 1e4, 3.0) if rot else qk, eps)
    page, row = table.cpu().numpy()[seq, pos // 64], pos % 64
    for got, want in ((qd.view(T, H, dk), qk[:, :H]), (kc[page, :, row], qk[:, H:]), (vc[page, :, row], x[:, (H + G) * dk:].reshape(T, G, dv))):
        off = np.abs(got.float().cpu().numpy() - want)
        assert (off < 3e-6 + (0 if dtype == torch.float32 else 2.0 ** -8 * np.abs(want))).all()
    assert int(err.item()) == 0 and int((kc != 0).any(-1).any(1).sum()) == T
