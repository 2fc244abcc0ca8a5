"""The recurrences by chunks (csrc/chunk_scan.cu) against the recurrence in float64: chunk edges, short sequences beside long ones,
every head size class, scratch that holds only a part of the step, and which calls take this route."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")
# As for the kernels that walk token by token (float32 state and sums): 2e-5 of the largest value.
TOL = 2e-5
# By chunks, the norm of the difference over the norm: 1.6e-7 at most over these cases.  An operand that lost its third bfloat16 term
# would be off by 2^-18 / sqrt(3) of itself on average, 1.3e-6 of the shorter or longer part of the sums that it enters.
CLOSE = 4e-7


def _ops():
    from longbow_quarrel_b200.kernels import ops
    return ops


def _i32(x):
    return torch.tensor(np.asarray(x), dtype=torch.int32, device=DEV)


def _scan64(q, k, v, a, b, S):
    """All [T, H, ...] float64; a [T, H, 1 or dk], b [T, H, 1]; returns outputs and the last state."""
    out = []
    for t in range(q.shape[0]):
        S = a[t][..., None] * S + (b[t] * k[t])[..., None] * v[t][:, None]
        out.append((S * q[t][..., None]).sum(1))
    return torch.stack(out), S


def _case(kind, lens, H, dk, dv, pad=0, seed=0, spoil=None):
    """A step's rows, the call's options and the float64 result.  spoil = (row, what): a number of that row that is not finite."""
    bad = lambda what: spoil is not None and spoil[1] == what
    gen = torch.Generator().manual_seed(seed + dk * dv)
    T, X = sum(lens), int(kind == "mlstm")
    x = torch.randn(T, 2 * H * dk + H * dv + pad, generator=gen).to(torch.bfloat16)
    if bad("v"):
        x[spoil[0], 2 * H * dk + 3] = float("inf")
    if bad("k"):
        x[spoil[0], H * dk + 3] = float("nan")
    slots = [2 * i + 1 for i in range(len(lens))][::-1]
    state = torch.randn(2 * len(lens) + 1, H, dk + X, dv + X, generator=gen)
    pos = np.concatenate([np.arange(n) + 3 * i for i, n in enumerate(lens)])
    opts, a, b, last_m = {}, None, torch.ones(T, H, 1, dtype=torch.float64), None
    z = x.double()
    q, k, v = z[:, :H * dk].view(T, H, dk), z[:, H * dk:2 * H * dk].view(T, H, dk), z[:, 2 * H * dk:2 * H * dk + H * dv].view(T, H, dv)
    if kind == "rotated":
        f = 1000.0 ** (-2.0 * torch.arange(dk // 2, dtype=torch.float64) / dk)
        ang = torch.arange(int(pos.max()) + 1, dtype=torch.float64)[:, None] * f[None]
        cos, sin = torch.cos(ang).float(), torch.sin(ang).float()
        opts["rot"] = (cos.to(DEV), sin.to(DEV), dk)
        c, s = cos.double()[pos][:, None], sin.double()[pos][:, None]
        turn = lambda y: torch.cat([y[..., :dk // 2] * c - y[..., dk // 2:] * s, y[..., dk // 2:] * c + y[..., :dk // 2] * s], -1)
        q, k = turn(q), turn(k)
    opts["q_scale"], opts["k_scale"] = dk ** -0.5, 0.5
    q, k = q * opts["q_scale"], k * opts["k_scale"]
    if kind == "mlstm":
        state[:, :, dk] = state[:, :, dk, :1]
        cap = 8.0
        pre, bias = torch.randn(T, 2 * H, generator=gen) * 2 * cap, torch.randn(2 * H, generator=gen)
        pre[T // 2:T // 2 + 5, H:] = -4 * cap                 # forget nearly everything
        if bad("gate") or bad("forget"):
            pre[spoil[0], 1 if bad("gate") else H + 1] = float("nan")
        opts["gates"] = (pre.to(DEV), bias.to(DEV), cap)
        g = pre.double() + bias.double()
        li, lf = cap * torch.tanh(g[:, :H] / cap), torch.nn.functional.logsigmoid(cap * torch.tanh(g[:, H:] / cap))
        v = torch.cat([v, torch.ones_like(v[..., :1])], dim=2)
    elif kind == "channels":
        # Decays from almost nothing kept to exactly one, in every mixture; a stretch that forgets all in the middle.
        pre = torch.randn(T, H * dk + 3, generator=gen)[:, 1:1 + H * dk] * 6
        pre[T // 3:T // 3 + 3] = -60.0
        bias, tau = torch.randn(H * dk, generator=gen) * 2, 2.0
        bias[::5], bias[1::7] = 60.0, -12.0
        if bad("decay"):
            pre[spoil[0], 5] = float("nan")
        dev = torch.zeros(T, H * dk + 3, device=DEV)
        dev[:, 1:1 + H * dk] = pre.to(DEV)
        opts["channel_decay"] = (dev[:, 1:1 + H * dk], bias.to(DEV), tau)
        a = torch.exp(torch.nn.functional.logsigmoid(pre.double() + bias.double()) / tau).view(T, H, dk)
    else:
        decay = torch.linspace(0.5, 1.0, H)
        opts["decay"] = decay.to(DEV)
        a = decay.double()[None, :, None].expand(T, H, 1)
    outs, finals, row = [], [], 0
    for n, slot in zip(lens, slots):
        S, rows = state[slot].double(), slice(row, row + n)
        if kind == "mlstm":
            m, aa, bb = S[:, dk, 0], [], []
            for t in range(row, row + n):
                m, old = torch.fmax(lf[t] + m, li[t]), m                # (the kernels' maxima pass a NaN gate over)
                aa.append(torch.exp(lf[t] + old - m)[:, None])
                bb.append(torch.exp(li[t] - m)[:, None])
            o, S = _scan64(q[rows], k[rows], v[rows], torch.stack(aa), torch.stack(bb), S[:, :dk])
            S = torch.cat([S, m[:, None, None].expand(-1, 1, dv + 1)], dim=1)
        else:
            o, S = _scan64(q[rows], k[rows], v[rows], a[rows], b[rows], S)
        outs.append(o)
        finals.append(S)
        row += n
    return x, state, slots, pos, opts, torch.cat(outs), finals


def _run(ops, x, state, slots, lens, pos, opts, H, dk, dv, known=None):
    before = ops.launches_by_name().get("linear_scan:chunks", 0)
    st = state.to(DEV).contiguous()
    out, enm = ops.linear_scan(x.to(DEV), 0, H * dk, 2 * H * dk, st, _i32(np.concatenate([[0], np.cumsum(lens)])), _i32(slots), _i32(pos),
                               len(lens), H, dk, dv, **opts, lens=known)
    return out.cpu().double(), st.cpu(), ops.launches_by_name().get("linear_scan:chunks", 0) - before


def _close(got, st, want, finals, slots):
    assert float((got - want).norm()) < CLOSE * float(want.norm())
    for slot, S in zip(slots, finals):
        assert float((st[slot].double() - S).norm()) < CLOSE * float(S.norm())


def _check(got, st, want, finals, state, slots):
    assert float((got - want).abs().max()) < TOL * float(want.abs().max())
    for slot, S in zip(slots, finals):
        assert float((st[slot].double() - S).abs().max()) < TOL * float(S.abs().max())
    others = [i for i in range(state.shape[0]) if i not in slots]
    assert torch.equal(st[others], state[others])


SIZES = [([64], 2, 64, 64), ([65, 1, 200], 3, 128, 128), ([191], 1, 16, 8), ([127, 130], 2, 64, 128), ([300, 2, 64], 2, 128, 40), ([129], 2, 80, 96)]


@pytest.mark.parametrize("lens,H,dk,dv", SIZES)
@pytest.mark.parametrize("kind", ["plain", "rotated", "mlstm", "channels"])
def test_chunks_follow_the_recurrence(kind, lens, H, dk, dv, monkeypatch):
    ops = _ops()
    monkeypatch.setattr(ops, "CHUNK_SCAN_ROWS_CHANNELS", ops.CHUNK_SCAN_ROWS)      # short sequences as well
    x, state, slots, pos, opts, want, finals = _case(kind, lens, H, dk, dv, pad=8)
    got, st, chunks = _run(ops, x, state, slots, lens, pos, opts, H, dk, dv)
    assert chunks == 1
    _check(got, st, want, finals, state, slots)
    _close(got, st, want, finals, slots)


@pytest.mark.parametrize("kind", ["plain", "mlstm", "channels"])
def test_scratch_for_a_part_of_the_chunks(kind, monkeypatch):
    """The chunks in turns of two places: the state goes on from turn to turn through its slot."""
    ops = _ops()
    lens, H, dk, dv = [200, 128, 130], 2, 64, 32
    x, state, slots, pos, opts, want, finals = _case(kind, lens, H, dk, dv)
    monkeypatch.setattr(ops, "CHUNK_SCRATCH_FLOATS", 2 * ops.build.load("chunk_scan").lq_chunk_place_floats(H, dk, dv, {"plain": 0, "mlstm": 1, "channels": 2}[kind]))
    got, st, chunks = _run(ops, x, state, slots, lens, pos, opts, H, dk, dv)
    assert chunks == 1
    _check(got, st, want, finals, state, slots)
    _close(got, st, want, finals, slots)


@pytest.mark.parametrize("kind", ["plain", "channels"])
@pytest.mark.parametrize("room", [3, 0])
def test_no_memory_for_the_scratch(kind, room, monkeypatch):
    """Room for three of the step's chunks: in turns, with the same bits.  For none: token by token."""
    ops = _ops()
    lens, H, dk, dv = [300, 140], 2, 64, 64
    x, state, slots, pos, opts, want, finals = _case(kind, lens, H, dk, dv)
    full, st_full, _ = _run(ops, x, state, slots, lens, pos, opts, H, dk, dv)
    most = room * ops.build.load("chunk_scan").lq_chunk_place_floats(H, dk, dv, {"plain": 0, "channels": 2}[kind])
    empty = torch.empty

    def limited(*size, **kw):
        if kw.get("dtype") == torch.float32 and size and isinstance(size[0], int) and size[0] > most:
            raise torch.cuda.OutOfMemoryError("test")
        return empty(*size, **kw)
    monkeypatch.setattr(torch, "empty", limited)
    got, st, chunks = _run(ops, x, state, slots, lens, pos, opts, H, dk, dv)
    monkeypatch.undo()
    assert chunks == int(room > 0)
    _check(got, st, want, finals, state, slots)
    assert not room or (torch.equal(got, full) and torch.equal(st, st_full))


@pytest.mark.parametrize("why,lens,H,dk,dv,pad", [("few rows", [63], 2, 64, 64, 0), ("odd head", [100], 2, 24, 20, 0), ("odd stride", [100], 2, 16, 16, 3),
                                                  ("a head of 136", [100], 1, 136, 16, 0)])
def test_other_sizes_keep_the_walk_by_tokens(why, lens, H, dk, dv, pad):
    ops = _ops()
    x, state, slots, pos, opts, want, finals = _case("plain", lens, H, dk, dv, pad=pad)
    got, st, chunks = _run(ops, x, state, slots, lens, pos, opts, H, dk, dv)
    assert chunks == 0
    _check(got, st, want, finals, state, slots)


@pytest.mark.parametrize("kind,what", [("plain", "v"), ("plain", "k"), ("rotated", "v"), ("mlstm", "v"), ("mlstm", "gate"), ("mlstm", "forget"), ("channels", "v"),
                                       ("channels", "decay"), ("channels", "k")])
@pytest.mark.parametrize("dk,dv,row", [(64, 64, 0), (64, 64, 13), (128, 128, 63), (64, 128, 85), (128, 64, 190)])
def test_a_number_that_is_not_finite_spoils_only_later_tokens(kind, what, dk, dv, row, monkeypatch):
    """A NaN (an infinity as a value) at one token of the first of two sequences: the same numbers are finite as in the recurrence, and those that
    are agree with it."""
    ops = _ops()
    monkeypatch.setattr(ops, "CHUNK_SCAN_ROWS_CHANNELS", ops.CHUNK_SCAN_ROWS)
    lens, H = [200, 70], 2
    x, state, slots, pos, opts, want, finals = _case(kind, lens, H, dk, dv, spoil=(row, what))
    got, st, chunks = _run(ops, x, state, slots, lens, pos, opts, H, dk, dv)
    assert chunks == 1
    fine = torch.isfinite(want)
    assert torch.equal(torch.isfinite(got), fine) and not fine[row:200].all() and fine[:row].all() and fine[200:].all()
    assert float((got - want)[fine].abs().max()) < TOL * float(want[fine].abs().max())
    for slot, S in zip(slots, finals):
        # Behind a NaN forget gate the kernels' running maximum (row dk) starts anew, a chunk's end later than the recurrence's.
        held, S = (st[slot][:, :dk].double(), S[:, :dk]) if what == "forget" else (st[slot].double(), S)
        fine = torch.isfinite(S)
        assert torch.equal(torch.isfinite(held), fine)
        if fine.any():
            assert float((held - S)[fine].abs().max()) < TOL * float(S[fine].abs().max())


@pytest.mark.parametrize("kind", ["plain", "rotated", "mlstm", "channels"])
@pytest.mark.parametrize("lens", [[400] + [1] * 7, [1, 63, 200, 5], [20, 30], [95, 97, 191, 193]])
@pytest.mark.parametrize("dk", [64, 32])
def test_a_sequence_takes_its_form_by_its_own_rows(kind, lens, dk):
    """Long sequences by chunks and short ones token by token in one step, whether the host knows their lengths or not; every sequence has
    the bits that it has alone."""
    ops = _ops()
    H, dv = 2, 64
    fewest = ops.chunk_scan_rows(dk, kind == "mlstm", kind == "channels")
    x, state, slots, pos, opts, want, finals = _case(kind, lens, H, dk, dv)
    got, st, chunks = _run(ops, x, state, slots, lens, pos, opts, H, dk, dv, known=lens)
    assert chunks == int(max(lens) >= fewest)
    _check(got, st, want, finals, state, slots)
    blind, st2, _ = _run(ops, x, state, slots, lens, pos, opts, H, dk, dv)
    assert torch.equal(blind, got) and torch.equal(st2, st)
    row = 0
    for n, slot in zip(lens, slots):
        rows = slice(row, row + n)
        own = dict(opts)
        if kind == "mlstm":
            own["gates"] = (opts["gates"][0][rows].contiguous(), *opts["gates"][1:])
        if kind == "channels":
            own["channel_decay"] = (opts["channel_decay"][0][rows], *opts["channel_decay"][1:])
        alone, st3, chunks = _run(ops, x[rows], state, [slot], [n], pos[rows], own, H, dk, dv, known=[n])
        assert chunks == int(n >= fewest)
        assert torch.equal(alone, got[rows]) and torch.equal(st3[slot], st[slot])
        row += n
