"""Recurrences that do not run token by token.

The linear attentions' recurrence with a request's tokens cut into segments that run side by side (csrc/linear_attention.cu)
against the recurrence token by token in float64: requests that end on, before and behind a segment's border, two steps
with the state carried over, decays from nearly nothing to a hair below one.

Tolerance: an output sums up to D * (tokens the decays let live) float32 products, in either order; 2e-5 of the row's
largest possible sum (the same recurrence over absolute values) holds at these sizes with room for 170 roundings."""
import pytest
import torch

gpu = pytest.mark.gpu
CASES = [  # heads, D, Dv, decay per head, tokens of the requests in the first and in the second step
    (2, 64, 128, False, (256,), (300,)), (3, 32, 96, False, (128, 129, 1), (257, 1, 127)), (1, 128, 64, False, (1, 700), (383, 1)),
    (2, 4, 4, True, (640, 0, 5), (0, 255, 130)), (4, 64, 128, True, (1000, 300), (128, 256)), (1, 100, 36, True, (511,), (513,)),
    (2, 96, 200, False, (300, 2), (0, 401)),
]


def plain(q, k, v, a, S):
    o = torch.zeros(q.shape[0], q.shape[1], v.shape[-1], dtype=torch.float64)
    for t in range(q.shape[0]):
        S = a[t][:, :, None] * S + k[t][:, :, None] * v[t][:, None, :]
        o[t] = (S * q[t][:, :, None]).sum(1)
    return o, S


@gpu
@pytest.mark.parametrize("heads,D,Dv,per_head,first,second", CASES)
def test_segments_against_token_by_token(heads, D, Dv, per_head, first, second):
    from airun_b200.engine.batch import Workspace
    from airun_b200.kernels import ops
    g = torch.Generator().manual_seed(heads * 1000 + D)
    slots = list(range(len(first) + 1))[::-1][:len(first)]
    state = torch.zeros(len(first) + 1, heads, D, Dv, device="cuda")
    want_state = [torch.zeros(heads, D, Dv, dtype=torch.float64) for _ in first]
    bound_state = [s.clone() for s in want_state]
    head_decay = torch.tensor([1.0 - 2.0 ** -(1 + 5 * h % 11) for h in range(heads)]).cuda()
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    ws = Workspace(torch.device("cuda"), 8 << 20)
    for lens in (first, second):
        T = sum(lens)
        row = 2 * heads * D + heads * Dv
        proj = torch.randn(T, row + 8, generator=g)
        decay = torch.rand(T, heads * D, generator=g) ** (0.02 + torch.rand(heads * D, generator=g) ** 4 * 3)
        decay[:, ::7] = 1e-20 ** torch.rand(T, (heads * D + 6) // 7, generator=g)
        pd = proj.cuda()
        q, k, v = pd[:, :heads * D], pd[:, heads * D:2 * heads * D], pd[:, 2 * heads * D:row]
        out = torch.empty(T, heads * Dv, device="cuda")
        cu = torch.tensor([sum(lens[:i]) for i in range(len(lens) + 1)], dtype=torch.int32, device="cuda")
        sl = torch.tensor(slots, dtype=torch.int32, device="cuda")
        assert ops._gla_work(ws, T, len(lens), heads, D, Dv, state)[1] > 0            # this is the cut form
        if per_head:
            ops.decay_recurrent(q, k, v, head_decay, True, state, cu, sl, len(lens), out, heads, D, Dv, 0.5, err, ws=ws)
        else:
            ops.gla_recurrent(q, k, v, decay.cuda(), state, cu, sl, len(lens), out, heads, D, Dv, 0.5, err, ws=ws)
        assert int(err.item()) == 0
        x = torch.nn.functional.silu(proj.double()) if per_head else proj.double()
        at = 0
        for r, n in enumerate(lens):
            rows = x[at:at + n]
            qq, kk, vv = (t.reshape(n, heads, w) for t, w in ((rows[:, :heads * D], D), (rows[:, heads * D:2 * heads * D], D), (rows[:, 2 * heads * D:row], Dv)))
            aa = head_decay.cpu().double()[None, :, None].expand(n, heads, D) if per_head else decay[at:at + n].double().reshape(n, heads, D)
            o, want_state[r] = plain(qq, kk, vv, aa, want_state[r])
            most, bound_state[r] = plain(qq.abs(), kk.abs(), vv.abs(), aa, bound_state[r])
            if n:
                got = out[at:at + n].cpu().double().reshape(n, heads, Dv)
                assert bool(((got - 0.5 * o).abs() <= 2e-5 * 0.5 * most + 1e-30).all())
            assert bool(((state[slots[r]].cpu().double() - want_state[r]).abs() <= 2e-5 * bound_state[r] + 1e-30).all())
            at += n
    assert float(state[[s for s in range(len(first) + 1) if s not in slots]].abs().max()) == 0


# ----------------------------------------------------------------------------- chunks of eight tokens, a decay per channel
CHUNK_CASES = [  # heads, q/k heads, D, Dv, tokens of the requests in the first and in the second step
    (2, 1, 64, 128, (140, 7), (1, 190)), (3, 3, 32, 20, (200, 9, 16), (15, 0, 223)), (1, 1, 128, 33, (77,), (64,)),
    (4, 2, 12, 8, (150, 3), (5, 130)), (2, 2, 100, 64, (1, 150), (133, 2)), (1, 1, 7, 5, (90,), (71,)), (2, 1, 128, 128, (257,), (130,)),
    (1, 1, 33, 16, (65, 64), (8, 121))]


@gpu
@pytest.mark.parametrize("mix", [False, True])
@pytest.mark.parametrize("heads,kv,D,Dv,first,second", CHUNK_CASES)
def test_chunks_with_a_decay_per_channel(heads, kv, D, Dv, first, second, mix):
    """The delta rule and the time mix in chunks (csrc/recurrent_state.cu) over two steps and then one token each, against token by token in float64;
    decays from 1e-20 to a hair below one.  Tolerance: unit keys and beta in (0, 1) let no error grow in the delta rule,
    each token adds a few roundings of the state's size, 2e-5 of the largest entry so far; the time mix as above."""
    import plain_pogarax as P
    from test_pirerax import batch_ctx
    from airun_b200.kernels import ops
    if mix:
        kv, Dv = heads, D
    g = torch.Generator().manual_seed(heads + 10 * D)
    slots = list(range(len(first) + 1))[::-1][:len(first)]
    n_state = heads * D * Dv
    state = torch.zeros(len(first) + 1, n_state + 4, device="cuda")
    want_state = [torch.zeros(heads, D, Dv, dtype=torch.float64) for _ in first]
    bonus = torch.randn(heads, D, generator=g)
    ends = [0] * len(first)
    for lens in (first, second, [1] * len(first)):
        live = [r for r, n in enumerate(lens) if n]
        ctx = batch_ctx([(ends[r], ends[r] + lens[r]) for r in live], [slots[r] for r in live])
        T = ctx.num_tokens
        q, k = (torch.nn.functional.normalize(torch.randn(T, kv, D, generator=g), dim=-1) for _ in range(2))
        v, beta = torch.randn(T, heads, Dv, generator=g), torch.randn(T, heads, generator=g)
        decay = torch.rand(T, heads, D, generator=g) ** (0.02 + torch.rand(heads, D, generator=g) ** 4 * 3)
        decay[:, :, ::5] = 1e-20 ** torch.rand(T, heads, (D + 4) // 5, generator=g)
        out = torch.empty(T, heads * Dv, device="cuda")
        args = [t.reshape(T, -1).cuda() for t in (q, k, v, decay)]
        if mix:
            ops.recurrent_state(ops.RECURRENCE_WKV, *args, state, ctx, out, heads, 1, D, Dv, bonus=bonus.cuda())
        else:
            ops.recurrent_state(ops.RECURRENCE_DELTA, *args, state, ctx, out, heads, heads // kv, D, Dv, beta=beta.cuda())
        assert int(ctx.err.item()) == 0
        at = 0
        for r in live:
            rows = slice(at, at + lens[r])
            qq, kk = (t[rows].double().repeat_interleave(heads // kv, dim=1) for t in (q, k))
            if mix:
                o, S = P.plain_wkv_recurrence(qq, kk, v[rows].double(), decay[rows].double(), bonus.double(), state=want_state[r])
            else:
                o, S = P.plain_delta_recurrence(qq, kk, v[rows].double(), decay[rows].double(), torch.sigmoid(beta[rows].double()), state=want_state[r])
            want_state[r] = S
            size = max(1.0, float(S.abs().max()), float(o.abs().max()))
            assert float((out[rows].cpu().double().view(-1, heads, Dv) - o).abs().max()) < 2e-5 * size
            assert float((state[slots[r], :n_state].cpu().double().view(heads, D, Dv) - S).abs().max()) < 2e-5 * size
            ends[r] += lens[r]
            at += lens[r]
    assert float(state[:, n_state:].abs().max()) == 0


@gpu
@pytest.mark.parametrize("per_head", [False, True])
def test_more_segments_than_were_made_room_for(per_head, monkeypatch):
    """A launch for fewer segments than the step has says so instead of leaving the rest out in silence."""
    from airun_b200.engine.batch import Workspace
    from airun_b200.kernels import ops
    heads, D, Dv, lens = 2, 32, 32, (300, 257)
    T, n = sum(lens), 3 + 3
    proj = torch.randn(T, 2 * heads * D + heads * Dv).cuda()
    q, k, v = proj[:, :heads * D], proj[:, heads * D:2 * heads * D], proj[:, 2 * heads * D:]
    cu, sl = torch.tensor([0, 300, T], dtype=torch.int32, device="cuda"), torch.arange(2, dtype=torch.int32, device="cuda")
    ws, true = Workspace(torch.device("cuda"), 8 << 20), ops._gla_work
    assert ops.segment_tokens() == 128
    for room, bits in ((n, 0), (n + 5, 0), (n - 1, 16), (1, 16)):
        monkeypatch.setattr(ops, "_gla_work", lambda *a, room=room: (true(*a)[0], room))
        state, out, err = torch.zeros(2, heads, D, Dv, device="cuda"), torch.empty(T, heads * Dv, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
        if per_head:
            ops.decay_recurrent(q, k, v, torch.full((heads,), 0.9, device="cuda"), False, state, cu, sl, 2, out, heads, D, Dv, 1.0, err, ws=ws)
        else:
            ops.gla_recurrent(q, k, v, torch.full((T, heads * D), 0.9, device="cuda"), state, cu, sl, 2, out, heads, D, Dv, 1.0, err, ws=ws)
        assert int(err.item()) == bits


def test_rules_count_the_portions_that_are_there():
    """A padded step names the requests its runner can hold; the rules go by the portions its graph is made for."""
    from types import SimpleNamespace

    from airun_b200.kernels import ops
    assert ops.portions_of(SimpleNamespace(num_reqs=64, extras={"device_plan": dict(max_rows=8, min_rows=1, max_portions=4)})) == 4
    assert ops.portions_of(SimpleNamespace(num_reqs=2, extras={"device_plan": dict(max_rows=0, min_rows=0, max_portions=4)})) == 2
    assert ops.portions_of(SimpleNamespace(num_reqs=3, extras={}, query_lens=[1, 700, 2])) == 2
    assert ops.portions_of(SimpleNamespace(num_reqs=5)) == 5
    assert ops.requests_of(SimpleNamespace(num_reqs=64, extras={"device_plan": dict(max_rows=8, min_rows=1, max_portions=4)})) == 12
    assert ops.requests_of(SimpleNamespace(num_reqs=10, extras={"device_plan": dict(max_rows=8, min_rows=1, max_portions=4)})) == 10
    assert ops.requests_of(SimpleNamespace(num_reqs=3, extras={}, query_lens=[1, 700, 2])) == 3


@gpu
@pytest.mark.parametrize("mode", ["channel", "mix", "head"])
def test_a_prompt_takes_the_same_form_whatever_its_runner_can_hold(mode):
    """One prompt in a step padded to 2 requests and to 64: the same bits, so the same kernels."""
    from types import SimpleNamespace

    from airun_b200.engine.batch import Workspace
    from airun_b200.kernels import ops
    g = torch.Generator().manual_seed(9)
    T, heads, D, Dv = 256, 2, 64, 64
    q, k, v = ((torch.randn(T, heads * D, generator=g) * 0.1).cuda() for _ in range(3))
    decay, beta = (torch.rand(T, heads * D, generator=g) ** 0.1).cuda(), torch.randn(T, heads, generator=g).cuda()
    outs = []
    for held in (2, 64):
        cu = torch.full((held + 1,), 230, dtype=torch.int32)
        cu[0] = 0
        ctx = SimpleNamespace(num_reqs=held, cu_tokens=cu.cuda(), state_slots=torch.arange(held, dtype=torch.int32).cuda(),
                              err=torch.zeros(1, dtype=torch.int32, device="cuda"), ws=Workspace(torch.device("cuda"), 8 << 20),
                              extras={"device_plan": dict(max_rows=0, min_rows=0, max_portions=1)})
        state, out = torch.zeros(held, heads * D * Dv, device="cuda"), torch.zeros(T, heads * Dv, device="cuda")
        if mode == "channel":
            ops.recurrent_state(ops.RECURRENCE_DELTA, q, k, v, decay, state, ctx, out, heads, 1, D, Dv, beta=beta)
        elif mode == "mix":
            ops.recurrent_state(ops.RECURRENCE_WKV, q, k, v, decay, state, ctx, out, heads, 1, D, Dv, bonus=beta[:heads].new_ones(heads, D))
        else:
            ops.recurrent_state(ops.RECURRENCE_DELTA_HEAD, q, k, v, beta, state, ctx, out, heads, 1, D, Dv, beta=beta,
                                a_log=beta.new_zeros(heads), dt_bias=beta.new_zeros(heads))
        used = ctx.ws.bytes() and ctx.ws.off
        assert int(ctx.err.item()) == 0
        outs.append((out[:230].clone(), state[0].clone(), used))
    assert torch.equal(outs[0][0], outs[1][0]) and torch.equal(outs[0][1], outs[1][1])
    assert outs[0][2] == outs[1][2] > 0                                  # coefficients were made: both ran in chunks


@gpu
@pytest.mark.parametrize("mode", ["channel", "mix", "head"])
@pytest.mark.parametrize("D,Dv,lens", [(64, 128, (203, 9)), (64, 40, (70, 131, 8)), (20, 33, (222,)), (32, 16, (65, 130))])
def test_chunks_of_two_columns_a_thread(mode, D, Dv, lens):
    """Enough heads that a thread takes two value columns, against the same heads in parts small enough for one: the sums are formed in the same
    order, so results and states differ by the roundings of contracted multiply-adds at most (2e-6 of the largest entry)."""
    from test_pirerax import batch_ctx
    from airun_b200.kernels import fast, ops
    Dv = D if mode == "mix" else Dv
    sms = fast.machine().sms
    n_part = 1 + max(1, sms // (len(lens) * -(-Dv // 16)))
    heads = 4 * n_part
    assert len(lens) * heads * -(-Dv // 16) > 2 * sms >= len(lens) * n_part * -(-Dv // 16)
    g = torch.Generator().manual_seed(D + Dv)
    T = sum(lens)
    q, k = (torch.nn.functional.normalize(torch.randn(T, heads, D, generator=g), dim=-1) for _ in range(2))
    v, beta = torch.randn(T, heads, Dv, generator=g), torch.randn(T, heads, generator=g)
    decay = torch.rand(T, heads, D, generator=g) ** 0.05
    start = torch.randn(len(lens), heads, D, Dv, generator=g)

    def run(lo, hi):
        n = hi - lo
        ctx = batch_ctx([(0, t) for t in lens], list(range(len(lens))))
        state, out = start[:, lo:hi].reshape(len(lens), -1).cuda(), torch.empty(T, n * Dv, device="cuda")
        flat = [t[:, lo:hi].reshape(T, -1).cuda() for t in (q, k, v, decay)]
        b = beta[:, lo:hi].contiguous().cuda()
        if mode == "channel":
            ops.recurrent_state(ops.RECURRENCE_DELTA, *flat, state, ctx, out, n, 1, D, Dv, beta=b)
        elif mode == "mix":
            ops.recurrent_state(ops.RECURRENCE_WKV, *flat, state, ctx, out, n, 1, D, Dv, bonus=b.new_ones(n, D))
        else:
            ops.recurrent_state(ops.RECURRENCE_DELTA_HEAD, *flat[:3], b, state, ctx, out, n, 1, D, Dv, beta=b, a_log=b.new_zeros(n), dt_bias=b.new_zeros(n))
        assert int(ctx.err.item()) == 0
        return out.view(T, n, Dv), state.view(len(lens), n, D, Dv)

    out, state = run(0, heads)
    for lo in range(0, heads, n_part):
        o, s = run(lo, lo + n_part)
        size = max(1.0, float(s.abs().max()), float(o.abs().max()))
        assert float((out[:, lo:lo + n_part] - o).abs().max()) <= 2e-6 * size and float((state[:, lo:lo + n_part] - s).abs().max()) <= 2e-6 * size
