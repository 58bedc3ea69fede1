"""Bananex on the GPU against the plain implementation (`plain_bananex.py`): every mechanism alone, whole and cut,
then whole models through the replayer in the four work splits, pages and slots used again, long decoding past
every window, and greedy generation through the entry point and its scheduler."""
import gc

import numpy as np
import pytest
import torch

import bananex_util as bu
import plain_bananex as pb
import replay_util as ru

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def rt32():
    from cuca_b200.runtime import Runtime
    return Runtime("cuda:0", torch.float32)


def _step(dev, portions, slots):
    """A hand-made step: request i brings rows `portions[i]` = (first position, count), in slot `slots[i]`."""
    from cuca_b200.engine.step import StepBatch
    pos, sor, row0, cnt, start = [], [], [], [], []
    for (p0, n), s in zip(portions, slots):
        row0.append(len(pos))
        pos += list(range(p0, p0 + n))
        sor += [s] * n
        cnt.append(n)
        start.append(p0)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=dev)  # noqa: E731
    return StepBatch(n_rows=len(pos), n_seqs=len(slots), tokens=None, positions=i32(pos), seq_of_row=i32(sor),
                     slots=i32(slots), logit_rows=None, n_logit_rows=0,
                     host={"counts": cnt, "slots": list(slots), "starts": start},
                     req_row0=i32(row0), req_count=i32(cnt), req_start=i32(start))


def _run_cut(dev, forward, inputs, cuts_per_request, slots, width):
    """Feed every request's rows of `inputs` (a list of [T_i, E] arrays) through `forward(h, step) -> [rows, width]`
    in steps that take the next cut of every request that still has one; returns the outputs per request."""
    done = [0] * len(inputs)
    outs = [[] for _ in inputs]
    k = 0
    while any(d < len(x) for d, x in zip(done, inputs)):
        who, portions, rows = [], [], []
        for i, x in enumerate(inputs):
            cuts = cuts_per_request[i]
            if done[i] < len(x) and k < len(cuts):
                n = min(cuts[k], len(x) - done[i])
                who.append(i)
                portions.append((done[i], n))
                rows.append(x[done[i]:done[i] + n])
        step = _step(dev, portions, [slots[i] for i in who])
        h = torch.tensor(np.concatenate(rows), dtype=torch.float32, device=dev)
        out = forward(h, step).cpu().numpy()
        r = 0
        for i, (_, n) in zip(who, portions):
            outs[i].append(out[r:r + n])
            done[i] += n
            r += n
        k += 1
    return [np.concatenate(o) for o in outs]


CUTS = [[1000], [1, 1, 1, 1, 1, 2, 3, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1000],
        [2, 5, 2, 16, 3, 2, 1, 1, 7, 1000]]


# ------------------------------------------------------------------------------------------ mechanisms alone
@pytest.mark.parametrize("P, N", [(64, 4), (64, 16), (70, 17), (64, 32), (20, 33), (64, 64), (33, 65), (8, 130), (130, 16)])
def test_state_scan_alone(rt32, P, N):
    """The state-space scan over every split of the state and its edges, single tokens beside portions longer than a run of
    staged tokens, from states that are not empty, against the recurrence in 64 bits; slots of no request stay."""
    from cuca_b200.kernels import ops
    dev, H, G = rt32.device, 4, 2
    g = torch.Generator(device=dev).manual_seed(P * N)
    counts, slots = [1, 40, 5, 17, 16], [3, 0, 5, 1, 2]
    rows = sum(counts)
    xbc = torch.randn(rows, H * P + 2 * G * N, device=dev, generator=g)
    proj = torch.randn(rows, H + 3, device=dev, generator=g)
    bias, a_log, skip = (torch.randn(H, device=dev, generator=g) for _ in range(3))
    state = torch.randn(6, H, P, N, device=dev, generator=g)
    got, y = state.clone(), torch.full((rows, H * P), 7.0, device=dev)
    ops.ssm_scan(xbc, proj, 2, bias, a_log, skip, got, y, _step(dev, [(0, n) for n in counts], slots), H, P, N, G)
    S, want, r = state.double(), torch.empty(rows, H, P, device=dev, dtype=torch.float64), 0
    for n, slot in zip(counts, slots):
        for _ in range(n):
            x = xbc[r, :H * P].double().view(H, P)
            B, C = (xbc[r, H * P + i * G * N:][:G * N].double().view(G, N).repeat_interleave(H // G, 0) for i in (0, 1))
            dt = torch.nn.functional.softplus(proj[r, 2:2 + H].double() + bias.double(), threshold=60)
            S[slot] = torch.exp(-torch.exp(a_log.double()) * dt)[:, None, None] * S[slot] + (dt[:, None] * x)[:, :, None] * B[:, None, :]
            want[r] = (S[slot] * C[:, None, :]).sum(-1) + skip.double()[:, None] * x
            r += 1
    assert (y.view_as(want).double() - want).abs().max() < 2e-5 * want.abs().max()
    assert (got.double() - S).abs().max() < 2e-5 * S.abs().max()
    assert torch.equal(got[4], state[4])


@pytest.mark.parametrize("P, N", [(64, 128), (20, 40), (64, 4)])
def test_state_scan_in_segments(rt32, P, N):
    """Long portions cut into runs that are walked side by side: against the recurrence in 64 bits, portions that end at,
    before and behind a run's end, in steps of several; portions of one run have the bits of the scan that cuts nothing, and
    a value that is no number stays with its request's later tokens."""
    from cuca_b200.kernels import ops
    dev, H, G = rt32.device, 4, 2
    run = int(__import__("cuca_b200.kernels.library", fromlist=["load"]).load().cuca_ssm_segment())
    g = torch.Generator(device=dev).manual_seed(P * N + 1)
    counts, slots = [1, run, run + 1, 2 * run, 2 * run + 301, 40], [3, 0, 5, 1, 2, 6]
    rows = sum(counts)
    xbc = torch.randn(rows, H * P + 2 * G * N, device=dev, generator=g)
    proj = torch.randn(rows, H + 3, device=dev, generator=g) - 2.0
    bias, a_log, skip = (torch.randn(H, device=dev, generator=g) for _ in range(3))
    state = torch.randn(7, H, P, N, device=dev, generator=g)
    step = _step(dev, [(0, n) for n in counts], slots)

    def scan(segments, x=xbc):
        st, y = state.clone(), torch.full((rows, H * P), 7.0, device=dev)
        ops.ssm_scan(x, proj, 2, bias, a_log, skip, st, y, step, H, P, N, G, segments=segments)
        return y, st
    y, got = scan(True)
    plain_y, plain = scan(False)
    r0 = 0
    for n, slot in zip(counts, slots):
        same = torch.equal(y[r0:r0 + n], plain_y[r0:r0 + n]) and torch.equal(got[slot], plain[slot])
        assert same == (n <= run), n
        S, r = state[slot].double(), r0
        xr = xbc[r:r + n, :H * P].double().view(n, H, P)
        B, C = (xbc[r:r + n, H * P + i * G * N:][:, :G * N].double().view(n, G, N).repeat_interleave(H // G, 1) for i in (0, 1))
        dt = torch.nn.functional.softplus(proj[r:r + n, 2:2 + H].double() + bias.double(), threshold=60)
        decay = torch.exp(-torch.exp(a_log.double()) * dt)
        want = torch.empty(n, H, P, device=dev, dtype=torch.float64)
        for t in range(n):
            S = decay[t][:, None, None] * S + (dt[t][:, None] * xr[t])[:, :, None] * B[t][:, None, :]
            want[t] = (S * C[t][:, None, :]).sum(-1) + skip.double()[:, None] * xr[t]
        assert (y[r0:r0 + n].view_as(want).double() - want).abs().max() < 2e-5 * want.abs().max(), n
        assert (got[slot].double() - S).abs().max() < 2e-5 * S.abs().max(), n
        r0 += n
    assert torch.equal(got[4], state[4])
    bad, at = xbc.clone(), sum(counts[:4]) + 100  # token 100 of the longest portion, the first head's first value
    bad[at, 0] = float("inf")
    z, zs = scan(True, bad)
    keep = torch.ones(rows, dtype=torch.bool, device=dev)
    keep[at:at + counts[4] - 100] = False
    assert torch.equal(z[keep], y[keep]) and not bool(z[~keep][:, 0].isfinite().any()) and not bool(zs[2, 0, 0].isfinite().all())


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("taps, C, rows", [(4, 4800, 130), (4, 300, 1700), (3, 4800, 530), (6, 4736, 514), (1, 4800, 530)])
def test_convolution_rows_are_the_same_bits_in_every_form(rt32, dtype, taps, C, rows):
    """So many rows and channels that a thread takes 16 rows, beside the same rows a few at a time (a thread a row), of
    requests whose borders lie anywhere; and against 64 bits."""
    from cuca_b200.kernels import ops
    dev = rt32.device
    g = torch.Generator(device=dev).manual_seed(C + taps)
    counts = [1, 2, 17, rows - 60, 3, 37]
    src = torch.randn(rows, C + 5, device=dev, generator=g)
    w, bias = (torch.randn(*s, device=dev, generator=g).to(dtype) for s in ((C, taps), (C,)))
    kept = torch.randn(len(counts), max(1, taps - 1), C, device=dev, generator=g)

    def run(portions, a, b, kept):
        out = torch.full((b - a, C), 7.0, device=dev)
        ops.causal_conv(src[a:b], 5, w, bias, kept, out, _step(dev, [(0, n) for _, n in portions], [s for s, _ in portions]))
        return out

    whole_kept = kept.clone()
    whole = run(list(enumerate(counts)), 0, rows, whole_kept)
    few_kept, a = kept.clone(), 0
    for i, n in enumerate(counts):
        pad = torch.cat([kept[i, :taps - 1], src[a:a + n, 5:]]).double()
        want = torch.nn.functional.silu(bias.double() + sum(w[:, k].double() * pad[k:k + n] for k in range(taps)))
        assert torch.allclose(whole[a:a + n].double(), want, atol=1e-5, rtol=1e-5)
        for b in range(0, n, 10):
            m = min(10, n - b)
            assert torch.equal(run([(i, m)], a + b, a + b + m, few_kept), whole[a + b:a + b + m]), (i, b)
        a += n
    assert torch.equal(few_kept[:, :taps - 1], whole_kept[:, :taps - 1])


@pytest.mark.parametrize("out_dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("H, N, K, T, o_pad", [(16, 512, 128, 300, 0), (40, 129, 40, 500, 3), (128, 100, 64, 130, 1)])
def test_head_contraction_rows_are_the_same_bits_in_every_form(rt32, out_dtype, H, N, K, T, o_pad):
    """So many rows that tiles of 128 are taken, beside the same rows 64 at a time (tiles of 64), with and without a gate, odd
    numbers of outputs and output strides among them; and against 64 bits."""
    from cuca_b200.kernels import ops
    dev = rt32.device
    g = torch.Generator(device=dev).manual_seed(N + T)
    a = torch.randn(T, H * (K + 4), device=dev, generator=g)
    w = torch.randn(H, N, K, device=dev, generator=g).to(torch.bfloat16)
    gate = torch.randn(T, H * N, device=dev, generator=g)

    def run(b, e, gate):
        out = torch.zeros(e - b, H * (N + o_pad), device=dev, dtype=out_dtype)
        ops.head_linear(a[b:e], a.stride(0), K + 4, w, out, out.stride(0), N + o_pad, e - b,
                        gate=None if gate is None else gate[b:e], ldg=H * N)
        return out

    for gt in (None, gate):
        whole = run(0, T, gt)
        for b in range(0, T, 64):
            e = min(T, b + 64)
            if e - b > 16:  # (16 rows and fewer are summed by warps, in another order)
                assert torch.equal(run(b, e, gt), whole[b:e]), b
        want = torch.einsum("thk,hnk->thn", a.view(T, H, K + 4)[:, :, :K].to(torch.bfloat16).double(), w.double())
        if gt is not None:
            want = want * torch.sigmoid(gt.double().view(T, H, N))
        got = whole.view(T, H, N + o_pad)
        tol = 1e-5 if out_dtype == torch.float32 else 2.0 ** -8
        assert torch.allclose(got[:, :, :N].double(), want, atol=tol * K ** 0.5, rtol=tol)
        assert bool((got[:, :, N:] == 0).all())



def test_norm_and_token_shift_alone(rt32):
    from cuca_b200.kernels import ops
    dev, E, eps = rt32.device, 52, 1e-5
    rs = np.random.default_rng(0)
    mix = rs.uniform(0, 1, E)
    gain = 1.3
    xs = [rs.normal(0, 2, (n, E)) for n in (23, 9)]
    want = [pb.token_shift(pb.rms(x, eps) * gain, mix) for x in xs]
    g = torch.tensor([gain], dtype=torch.float32, device=dev)
    m = torch.tensor(mix, dtype=torch.float32, device=dev)
    for cuts in ([CUTS[0], CUTS[0]], [CUTS[1], CUTS[2]], [CUTS[2], CUTS[1]]):
        kept = torch.zeros(4, E, device=dev)
        kept[0] = 7.0  # another request's row must stay as it is

        def fwd(h, step):
            out = torch.empty_like(h)
            ops.norm_shift(h, g, eps, m, kept, out, step)
            return out
        got = _run_cut(dev, fwd, xs, cuts, [2, 3], E)
        for a, b in zip(got, want):
            assert np.abs(a - b).max() < 1e-5
        assert torch.equal(kept[0].cpu(), torch.full((E,), 7.0))
    # a vector gain through the same kernel
    gv = rs.normal(1, 0.2, E)
    kept = torch.zeros(4, E, device=dev)
    out = torch.empty(23, E, device=dev)
    ops.norm_shift(torch.tensor(xs[0], dtype=torch.float32, device=dev), torch.tensor(gv, dtype=torch.float32, device=dev),
                   eps, m, kept, out, _step(dev, [(0, 23)], [1]))
    assert np.abs(out.cpu().numpy() - pb.token_shift(pb.rms(xs[0], eps) * gv, mix)).max() < 1e-5


def test_post_norm_add_alone(rt32):
    from cuca_b200.kernels import ops
    dev, E, eps = rt32.device, 70, 1e-6
    rs = np.random.default_rng(1)
    x, y = rs.normal(0, 1, (11, E)), rs.normal(0, 3, (11, E))
    xd = torch.tensor(x, dtype=torch.float32, device=dev)
    out = torch.empty(11, E, device=dev)
    g1, g2 = torch.tensor([0.8], device=dev), torch.tensor([1.7], device=dev)
    ops.post_norm_add(xd, torch.tensor(y, dtype=torch.float32, device=dev), g1, eps, gain2=g2, out=out)
    nx = x + pb.rms(y, eps) * 0.8
    assert np.abs(xd.cpu().numpy() - nx).max() < 1e-5
    assert np.abs(out.cpu().numpy() - pb.rms(nx, eps) * 1.7).max() < 1e-5


def _part(kind, cls, layer, rt, E, eps, prefix="l0.mix."):
    from cuca_b200.config.bananex_config import BananexConfig
    from cuca_b200.models.bananex import _mixer_spec
    cfg = BananexConfig.from_json(bu.config([layer], width=E, eps=eps))
    spec = _mixer_spec(cfg.layers[0], E, eps, prefix)
    assert spec.kind == kind
    return cls(spec, rt)


def _weights_for(part, seed):
    rs = np.random.default_rng(seed)
    ws = {}
    for name, need in part.tensors().items():
        shape = tuple(need.shape)
        if name.endswith("A_log"):
            v = rs.uniform(-1.5, 1.0, shape)
        elif name.endswith("dt_bias"):
            v = rs.uniform(-2, 1, shape)
        elif need.init == "ones" or name.endswith(".D"):
            v = 1 + rs.normal(0, 0.3, shape)
        elif len(shape) == 1:
            v = rs.normal(0, 0.3, shape)
        elif name.endswith(".conv"):
            v = rs.normal(0, 0.5, shape)
        else:
            v = rs.normal(0, 1, shape) / np.sqrt(shape[-1])
        ws[name] = np.asarray(v, dtype=np.float32).astype(np.float64)
    return ws


def _load(part, ws, dev):
    part.load(lambda n: torch.tensor(ws[n], dtype=torch.float32, device=dev))


@pytest.mark.parametrize("inner", [48, 130])
def test_mingru_alone_whole_and_cut(rt32, inner):
    from cuca_b200.parts.recurrent import MinGRU
    dev, E = rt32.device, 40
    part = _part("mingru", MinGRU, bu.mingru(inner), rt32, E, 1e-5)
    ws = _weights_for(part, 3)
    _load(part, ws, dev)
    rs = np.random.default_rng(4)
    xs = [rs.normal(0, 1.5, (n, E)) for n in (37, 12, 5)]
    want = [pb.mingru(x, ws, "l0.mix.", {"width": inner}) for x in xs]
    for cuts in ([CUTS[0]] * 3, [CUTS[1], CUTS[2], CUTS[1]], [CUTS[2], CUTS[1], CUTS[0]]):
        state = torch.zeros(4, inner, device=dev)

        def fwd(h, step):
            from cuca_b200.cache.device import CacheView
            out = torch.zeros(h.shape[0], E, device=dev)
            part.forward(h, out, step, CacheView(None, None, None, 16, -1, {"mingru": state}, step.slots))
            return out
        got = _run_cut(dev, fwd, xs, cuts, [3, 0, 2], E)
        for a, b in zip(got, want):
            assert np.abs(a - b).max() < 2e-5 * max(1.0, np.abs(b).max())


def test_mingru_long_portions_in_chunks():
    """In bfloat16 a portion of 256 tokens or more runs as chunks side by side with the state carried across
    them: whole, and cut so that a chunked portion starts from a state that single tokens left."""
    from cuca_b200.cache.device import CacheView
    from cuca_b200.kernels import ops
    from cuca_b200.parts.recurrent import MinGRU
    from cuca_b200.runtime import Runtime
    rt = Runtime("cuda:0", torch.bfloat16)
    dev, E, inner = rt.device, 40, 70
    part = _part("mingru", MinGRU, bu.mingru(inner), rt, E, 1e-5)
    ws = {k: bu.bf16_round(v) for k, v in _weights_for(part, 3).items()}
    part.load(lambda n: torch.tensor(ws[n], dtype=torch.bfloat16, device=dev))
    rs = np.random.default_rng(4)
    xs = [bu.bf16_round(rs.normal(0, 1.5, (n, E))) for n in (700, 300)]
    want = [pb.mingru(x, ws, "l0.mix.", {"width": inner}) for x in xs]
    assert ops.MINGRU_CHUNKED_FROM <= 256
    for cuts in ([CUTS[0]] * 2, [[1, 1, 3, 290, 1, 1, 1000], [260, 1, 1000]]):
        state = torch.zeros(4, inner, device=dev)

        def fwd(h, step):
            stream = rt.stream(torch.zeros(h.shape[0], E, device=dev))
            part.forward(h.to(torch.bfloat16), stream, step, CacheView(None, None, None, 16, -1, {"mingru": state}, step.slots))
            return stream.data
        got = _run_cut(dev, fwd, xs, cuts, [2, 1], E)
        for a, b in zip(got, want):
            assert np.abs(a - b).max() < 3e-2 * np.abs(b).max()


@pytest.mark.parametrize("layer", [bu.mamba2(), bu.mamba2(heads=3, vdim=20, state=40, groups=3, conv=1, norm_groups=3),
                                   bu.mamba2(heads=2, vdim=64, state=128, groups=1, conv=7, norm_groups=1),
                                   bu.mamba2(heads=4, vdim=12, state=6, groups=4, conv=2, norm_groups=4)])
def test_mamba2_alone_whole_and_cut(rt32, layer):
    from cuca_b200.parts.recurrent import Mamba2
    dev, E, eps = rt32.device, 44, 1e-5
    part = _part("mamba2", Mamba2, layer, rt32, E, eps)
    ws = _weights_for(part, 5)
    _load(part, ws, dev)
    rs = np.random.default_rng(6)
    xs = [rs.normal(0, 1.5, (n, E)) for n in (41, 3, 17)]
    want = [pb.mamba2(x, ws, "l0.mix.", layer["mixer"], eps) for x in xs]
    needs = part.cache_needs().state
    for cuts in ([CUTS[0]] * 3, [CUTS[1], CUTS[2], CUTS[1]], [CUTS[2], CUTS[1], CUTS[2]]):
        state = {k: torch.zeros(4, *v.shape, device=dev) for k, v in needs.items()}

        def fwd(h, step):
            from cuca_b200.cache.device import CacheView
            out = torch.zeros(h.shape[0], E, device=dev)
            part.forward(h, out, step, CacheView(None, None, None, 16, -1, state, step.slots))
            return out
        got = _run_cut(dev, fwd, xs, cuts, [1, 3, 0], E)
        for a, b in zip(got, want):
            assert np.abs(a - b).max() < 3e-5 * max(1.0, np.abs(b).max())


@pytest.mark.parametrize("layer", [bu.latent(window=12), bu.latent(window=None, dims=4),
                                   bu.latent(heads=1, dim=32, rot_dim=4, vdim=16, kv_rank=136, window=1),
                                   bu.latent(heads=5, dim=12, rot_dim=6, vdim=10, kv_rank=33, window=16, scale=1.2),
                                   bu.latent(heads=2, dim=8, rot_dim=16, vdim=8, kv_rank=300, window=33)])
def test_latent_attention_alone_whole_and_cut(rt32, layer):
    """Pages of 8 positions handed out in a scrambled order; windows of 1, 12, 16 (two pages exactly), 33 (one past
    four pages) and none; decoding one by one walks every window edge over page borders."""
    from cuca_b200.cache.device import CacheView
    from cuca_b200.parts.latent_attention import LatentAttention
    dev, E, eps, bs = rt32.device, 36, 1e-5, 8
    part = _part("latent_attention", LatentAttention, layer, rt32, E, eps)
    ws = _weights_for(part, 7)
    _load(part, ws, dev)
    part.prepare(128)
    rs = np.random.default_rng(8)
    xs = [rs.normal(0, 1.5, (n, E)) for n in (75, 20)]
    want = [pb.latent_attention(x, ws, "l0.mix.", layer["mixer"], eps) for x in xs]
    order = rs.permutation(16).tolist()
    for cuts in ([CUTS[0]] * 2, [CUTS[1], CUTS[2]], [CUTS[2], CUTS[1]]):
        pool = torch.full((16, 1, bs, part.key_dim), float("nan"), device=dev)
        tables = torch.full((4, 16), -1, dtype=torch.int32, device=dev)
        tables[2, :10] = torch.tensor(order[:10], dtype=torch.int32)
        tables[0, :3] = torch.tensor(order[10:13], dtype=torch.int32)

        def fwd(h, step):
            out = torch.zeros(h.shape[0], E, device=dev)
            part.forward(h, out, step, CacheView(pool, None, tables, bs, 0, None, step.slots))
            return out
        got = _run_cut(dev, fwd, xs, cuts, [2, 0], E)
        for a, b in zip(got, want):
            assert np.abs(a - b).max() < 2e-5 * max(1.0, np.abs(b).max())
    assert int(rt32.err.item()) == 0


@pytest.mark.parametrize("layer", [
    bu.latent(heads=3, dim=16, rot_dim=16, vdim=24, kv_rank=64, window=20, scale=1.0),
    bu.latent(heads=20, dim=8, rot_dim=32, vdim=8, kv_rank=96, window=None, scale=0.8),
    bu.latent(heads=2, dim=24, rot_dim=16, vdim=12, kv_rank=256, window=70, scale=0.9),
    bu.latent(heads=1, dim=8, rot_dim=64, vdim=8, kv_rank=512, window=130, scale=1.0),
    bu.latent(heads=16, dim=16, rot_dim=0, vdim=8, kv_rank=32, window=64, scale=1.0)])
def test_latent_attention_on_tensor_cores(layer):
    """The bfloat16 forms: prompts in groups of 16 tokens per head, single tokens with their heads as the group.
    Scales near one make the softmax pick few keys, so a key that is dropped, seen too early or too late moves
    the result by far more than rounding does. 200 tokens walk windows over several key tiles and page borders."""
    from cuca_b200.cache.device import CacheView
    from cuca_b200.kernels import ops
    from cuca_b200.parts.latent_attention import LatentAttention
    from cuca_b200.runtime import Runtime
    rt = Runtime("cuda:0", torch.bfloat16)
    dev, E, eps, bs = rt.device, 48, 1e-5, 16
    part = _part("latent_attention", LatentAttention, layer, rt, E, eps)
    assert ops.latent_attention_mma_supported(part.rank, part.key_dim)
    ws = {k: bu.bf16_round(v) for k, v in _weights_for(part, 11).items()}
    needs = part.tensors()
    part.load(lambda n: torch.tensor(ws[n], dtype=torch.float32 if needs[n].keep_fp32 else torch.bfloat16, device=dev))
    part.prepare(256)
    rs = np.random.default_rng(12)
    xs = [bu.bf16_round(rs.normal(0, 1.5, (n, E))) for n in (200, 37)]
    want = [pb.latent_attention(x, ws, "l0.mix.", layer["mixer"], eps) for x in xs]
    pb.ROUND = bu.bf16_round
    try:
        rounded = [pb.latent_attention(x, ws, "l0.mix.", layer["mixer"], eps) for x in xs]
    finally:
        pb.ROUND = None
    tol = [max(2e-2 * np.abs(b).max(), 4 * np.abs(a - b).max()) for a, b in zip(rounded, want)]
    order = rs.permutation(20).tolist()
    for cuts in ([CUTS[0]] * 2, [[150] + CUTS[1], CUTS[2]], [[3, 64, 17, 90] + CUTS[1], CUTS[1]]):
        pool = torch.full((20, 1, bs, part.key_dim), float("nan"), dtype=torch.bfloat16, device=dev)
        tables = torch.full((4, 16), -1, dtype=torch.int32, device=dev)
        tables[1, :13] = torch.tensor(order[:13], dtype=torch.int32)
        tables[3, :3] = torch.tensor(order[13:16], dtype=torch.int32)

        def fwd(h, step):
            stream = rt.stream(torch.zeros(h.shape[0], E, device=dev))  # few rows may leave slices pending on it
            part.forward(h.to(torch.bfloat16), stream, step, CacheView(pool, None, tables, bs, 0, None, step.slots))
            return stream.data
        got = _run_cut(dev, fwd, xs, cuts, [1, 3], E)
        for a, b, t in zip(got, want, tol):
            assert np.isfinite(a).all() and np.abs(a - b).max() < t, (np.abs(a - b).max(), t)
    assert int(rt.err.item()) == 0


@pytest.mark.parametrize("counts,cut", [([1] * 40 + [1985] + [1] * 23, [40]), ([600] * 66, list(range(64))),
                                        ([513, 1, 1537, 512, 40, 700], [0, 2, 5]), ([1, 1100, 1100], [1, 2])])
def test_state_scan_in_segments_beside_other_requests(rt32, counts, cut):
    """Scratch is for the segments there are, whatever else the step brings; whole walks and cut ones have the bits that they have
    alone. Of more portions than one launch holds, the first are cut."""
    from cuca_b200.kernels import library, ops
    dev, H, G, P, N = rt32.device, 4, 1, 64, 128
    run = int(library.load().cuca_ssm_segment())
    g = torch.Generator(device=dev).manual_seed(len(counts))
    rows, slots = sum(counts), list(range(len(counts)))[::-1]
    xbc = torch.randn(rows, H * P + 2 * G * N, device=dev, generator=g)
    proj = torch.randn(rows, H, device=dev, generator=g) - 2.0
    bias, a_log, skip = (torch.randn(H, device=dev, generator=g) for _ in range(3))
    state = torch.randn(len(counts), H, P, N, device=dev, generator=g)

    def scan(which, segments):
        first = [sum(counts[:q]) for q in which]
        at = torch.cat([torch.arange(f, f + counts[q], device=dev) for f, q in zip(first, which)])
        x, pr, st, y = xbc[at], proj[at], state.clone(), torch.full((len(at), H * P), 7.0, device=dev)
        step = _step(dev, [(0, counts[q]) for q in which], [slots[q] for q in which])
        gc.collect()  # (what earlier tests left in cycles must not be freed in between)
        before = torch.cuda.memory_allocated()
        torch.cuda.reset_peak_memory_stats()
        ops.ssm_scan(x, pr, 0, bias, a_log, skip, st, y, step, H, P, N, G, segments=segments)
        return y, st, torch.cuda.max_memory_allocated() - before
    everyone = list(range(len(counts)))
    y, st, scratch = scan(everyone, True)
    plain_y, plain, none = scan(everyone, 0)
    cells = sum(-(-counts[q] // run) for q in cut)
    assert none == 0 and scratch <= cells * H * (P * N + 1) * 4 + 512
    r = 0
    for q, n in enumerate(counts):
        same = torch.equal(y[r:r + n], plain_y[r:r + n]) and torch.equal(st[slots[q]], plain[slots[q]])
        assert same == (q not in cut), q
        if q in cut[:3]:
            alone_y, alone, _ = scan([q], True)
            assert torch.equal(y[r:r + n], alone_y) and torch.equal(st[slots[q]], alone[slots[q]])
        r += n


def test_state_scan_is_cut_where_it_leaves_the_gpu_empty(rt32):
    """One long portion, alone or beside single tokens; not short ones, not many, not sizes that take no segments."""
    from cuca_b200.kernels import ops
    dev = rt32.device

    def cut_from(counts, H=64, P=64, N=128):
        return ops.ssm_cut_from(_step(dev, [(0, n) for n in counts], list(range(len(counts)))), H, P, N)
    assert cut_from([2048]) == 1536 and cut_from([1985] + [1] * 63) == 1536 and cut_from([1535]) == 0 and cut_from([2048] * 4) == 0
    assert cut_from([1024], 24, 64, 64) == 1024 and cut_from([1023], 24, 64, 64) == 0
    assert cut_from([2048], 4, 66, 128) == 0 and cut_from([2048], 4, 64, 130) == 0 and cut_from([1]) == 0


@pytest.mark.parametrize("layer,tokens", [
    (bu.latent(heads=16, dim=8, rot_dim=64, vdim=8, kv_rank=512, window=130, scale=1.0), 8),  # two halves of the columns
    (bu.latent(heads=16, dim=16, rot_dim=0, vdim=8, kv_rank=64, window=None, scale=1.0), 8),  # one chunk of values
    (bu.latent(heads=8, dim=24, rot_dim=64, vdim=12, kv_rank=320, window=70, scale=0.9), 16),  # unequal parts of the columns
    (bu.latent(heads=24, dim=8, rot_dim=0, vdim=8, kv_rank=256, window=1, scale=0.8), 16),  # all queries in tensor memory
    (bu.latent(heads=32, dim=8, rot_dim=128, vdim=8, kv_rank=448, window=64, scale=1.0), 8)])  # two groups of heads
def test_latent_attention_in_groups_of_tokens_and_heads(layer, tokens):
    """The tcgen05 form's sizes through the test above: portions that end inside a group and inside a key tile, windows over
    several key tiles, pages that hold NaN where nothing was written."""
    from cuca_b200.kernels import ops
    m = layer["mixer"]
    assert ops.latent_attention_tc_tokens(m["heads"], m["kv_rank"], m["kv_rank"] + m["rot_dim"], m["scale"]) == tokens
    test_latent_attention_on_tensor_cores(layer)


@pytest.mark.parametrize("off", [0, 1])
@pytest.mark.parametrize("portions", [[(0, 40), (5, 2)], [(0, 70), (30, 34), (0, 64)]])
def test_latent_attention_of_operands_off_16_bytes_and_of_few_keys(off, portions):
    """Where the tcgen05 form does not take the addresses, or is not worth its start, the other tensor-core form runs. Against the
    plain kernel; queries and weights are bfloat16 numbers (2^-9), the values of a row at most their maximum."""
    from cuca_b200.cache.device import CacheView
    from cuca_b200.kernels import ops
    dev, H, rank, rot, bs = torch.device("cuda:0"), 8, 64, 64, 16
    Dk, n = rank + rot, sum(c for _, c in portions)
    g = torch.Generator(device=dev).manual_seed(n)
    step = _step(dev, portions, list(range(len(portions))))
    pool = torch.randn(32, 1, bs, Dk, device=dev, generator=g).to(torch.bfloat16)
    tables = torch.randperm(32, device=dev, generator=g).to(torch.int32)[:len(portions) * 8].view(-1, 8).contiguous()
    qk = torch.empty(n * H * Dk + off, device=dev)[off:].view(n, H, Dk).normal_(generator=g)
    cache, err, got = CacheView(pool, None, tables, bs, 0, None, step.slots), torch.zeros(1, dtype=torch.int32, device=dev), []
    for tensor_cores in (True, False):
        out = torch.full((n * H * rank + off,), 9.0, device=dev)[off:].view(n, H, rank)
        ops.USE_MMA_LATENT = tensor_cores
        try:
            ops.latent_attention(qk, out, cache, step, H, rank, Dk, 0.1, None, err)
        finally:
            ops.USE_MMA_LATENT = True
        got.append(out)
    assert int(err.item()) == 0 and (got[0] - got[1]).abs().max() < 2e-2 * got[1].abs().max()


def test_dense_feed_forward_and_loop_entry_alone(rt32):
    from cuca_b200.parts.base import PartSpec
    from cuca_b200.parts.mlp import DenseActivation
    from cuca_b200.parts.stream_ops import LoopEntry
    dev, E, F = rt32.device, 28, 50
    rs = np.random.default_rng(9)
    ff = DenseActivation(PartSpec("dense_act", {"width": E, "inner": F, "act": "gelu", "bias": True},
                                  {"up": "m.up", "up_bias": "m.up.b", "down": "m.down", "down_bias": "m.down.b"}), rt32)
    ws = {"m.up": rs.normal(0, 0.4, (F, E)), "m.up.b": rs.normal(0, 0.5, F), "m.down": rs.normal(0, 0.3, (E, F)),
          "m.down.b": rs.normal(0, 0.5, E)}
    _load(ff, ws, dev)
    h = rs.normal(0, 1.5, (13, E))
    out = torch.zeros(13, E, device=dev)
    ff.forward(torch.tensor(h, dtype=torch.float32, device=dev), out, None)
    assert np.abs(out.cpu().numpy() - pb.dense_ff(h, ws, "m.")).max() < 2e-5
    op = LoopEntry(PartSpec("loop_entry", {"width": E, "times": 3}, {"mix": "loop.in", "step": "loop.step"}), rt32)
    wl = {"loop.in": rs.normal(0, 0.3, (E, 2 * E)), "loop.step": rs.normal(0, 1, (3, E))}
    _load(op, wl, dev)
    x, e = rs.normal(0, 1, (13, E)), rs.normal(0, 1, (13, E))
    stream = rt32.stream(torch.tensor(x, dtype=torch.float32, device=dev))
    ed = torch.tensor(e, dtype=torch.float32, device=dev)
    op.forward(stream, ed, None, 2)
    assert np.abs(stream.data.cpu().numpy() - (np.concatenate([x, e], 1) @ wl["loop.in"].T + wl["loop.step"][2])).max() < 2e-5
    assert np.array_equal(ed.cpu().numpy(), e.astype(np.float32))  # the embedding output is only read


# ------------------------------------------------------------------------------------------ whole models
LENGTHS = {"wide": [1, 15, 16, 17, 63, 65, 140], "mix": [1, 2, 5, 16, 33, 64, 97, 130], "loop0": [3, 17, 48, 100], "flat": [2, 40, 41, 42, 90, 150],
           "once": [1, 18, 35, 77]}


@pytest.fixture(scope="module")
def models(tmp_path_factory):
    out = {}
    for i, (name, cfg) in enumerate(bu.CONFIGS.items()):
        weights = bu.make_weights(cfg, seed=20 + i)
        out[name] = (bu.write_model(tmp_path_factory.mktemp(f"bananex_{name}"), cfg, weights), cfg,
                     bu.Oracle(cfg, weights))
    return out


def _requests(name, cfg):
    return {f"r{n}": bu.random_tokens(n, cfg["vocab"], seed=300 + n) for n in LENGTHS[name]}


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("name", list(bu.CONFIGS))
def test_whole_and_decoded_one_by_one(models, name, dtype):
    folder, cfg, oracle = models[name]
    reqs = _requests(name, cfg)
    for steps in (ru.trace_whole(reqs), ru.trace_tail_one_by_one(reqs, tail=48)):
        got = ru.run_in_process(folder, dtype, steps, ru.peak_tokens(steps), block_size=8)
        ru.compare(steps, got, reqs, oracle, oracle.tolerance(dtype, reqs))


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("name", list(bu.CONFIGS))
def test_portions_down_to_two_tokens(models, name, dtype):
    folder, cfg, oracle = models[name]
    reqs = _requests(name, cfg)
    for sizes in ((5, 2, 17, 3, 2, 32, 7, 2, 64, 11), (2, 2, 3, 1, 1, 8, 9, 40)):
        steps = ru.trace_portions(reqs, sizes=sizes)
        got = ru.run_in_process(folder, dtype, steps, ru.peak_tokens(steps), block_size=16)
        ru.compare(steps, got, reqs, oracle, oracle.tolerance(dtype, reqs))


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("name", list(bu.CONFIGS))
def test_mixed_batches_reuse_pages_and_slots(models, name, dtype):
    """Eight and more requests through four (and three) slots and a pool sized for the peak: every slot and most
    pages serve several requests, whose state must start from zero; windowed groups give pages back as they go."""
    folder, cfg, oracle = models[name]
    reqs = _requests(name, cfg)
    reqs.update({f"s{n}": bu.random_tokens(n, cfg["vocab"], seed=900 + n) for n in (4, 9, 23, 31, 58)})
    for live, pools in ((4, "full"), (3, "sized")):
        steps = ru.trace_mixed(reqs, max_live=live, seed=7 + live)
        got = ru.run_in_process(folder, dtype, steps, ru.peak_tokens(steps), block_size=8, window_pools=pools)
        ru.compare(steps, got, reqs, oracle, oracle.tolerance(dtype, reqs))


def test_32_bit_does_not_depend_on_cuts_or_company(models):
    """In 32-bit a position's logits are the same bits whole, in portions, decoded and beside other requests."""
    folder, cfg, _ = models["mix"]
    reqs = {"a": bu.random_tokens(70, cfg["vocab"], 1), "b": bu.random_tokens(33, cfg["vocab"], 2)}
    whole = ru.trace_whole(reqs)
    ref = ru.run_in_process(folder, "float32", whole, ru.peak_tokens(whole))
    want = {rid: ref[i] for i, rid in enumerate(reqs)}
    for steps in (ru.trace_portions(reqs, sizes=(3, 2, 9, 1, 1, 30)), ru.trace_mixed(reqs, max_live=2, seed=3)):
        got = ru.run_in_process(folder, "float32", steps, ru.peak_tokens(steps))
        pos = {rid: 0 for rid in reqs}
        for s in steps:
            row = 0
            for e in s["entries"]:
                for w in e["want"]:
                    assert np.array_equal(got[s["step"]][row], want[e["id"]][pos[e["id"]] + w]), (s["step"], e["id"])
                    row += 1
                pos[e["id"]] += len(e["tokens"])


def test_long_decoding_past_every_window(models):
    folder, cfg, oracle = models["flat"]
    reqs = {"long": bu.random_tokens(230, cfg["vocab"], 5)}
    steps = ru.trace_tail_one_by_one(reqs, tail=200)
    for dtype in ("float32", "bfloat16"):
        got = ru.run_in_process(folder, dtype, steps, ru.peak_tokens(steps), block_size=8, window_pools="sized")
        ru.compare(steps, got, reqs, oracle, oracle.tolerance(dtype, reqs))


def test_long_prompts(models):
    """Prompts long enough for the forms that only long portions take (chunks of the gated recurrence side by side,
    many key tiles per group of the tensor-core attention), whole and in portions that start inside a chunk."""
    folder, cfg, oracle = models["wide"]
    reqs = {"p": bu.random_tokens(610, cfg["vocab"], 8), "q": bu.random_tokens(300, cfg["vocab"], 9)}
    for steps in (ru.trace_whole(reqs), ru.trace_portions(reqs, sizes=(7, 300, 2, 280, 1, 64))):
        for dtype in ("bfloat16", "float32"):
            got = ru.run_in_process(folder, dtype, steps, ru.peak_tokens(steps), block_size=16)
            ru.compare(steps, got, reqs, oracle, oracle.tolerance(dtype, reqs))


def test_trace_run_as_a_program(models):
    folder, cfg, oracle = models["loop0"]
    reqs = _requests("loop0", cfg)
    steps = ru.trace_mixed(reqs, max_live=4, seed=1)
    got = ru.run_subprocess(folder, "float32", steps, ru.peak_tokens(steps))
    ru.compare(steps, got, reqs, oracle, oracle.tolerance("float32", reqs))


# ------------------------------------------------------------------------------------------ the entry point
def _plain_greedy(cfg, w, prompt, n):
    toks = list(prompt)
    for _ in range(n):
        toks.append(int(np.argmax(pb.forward(cfg, w, toks)[-1])))
    return toks[len(prompt):]


@pytest.mark.parametrize("name", ["mix", "flat"])
def test_greedy_generation_through_the_entry_point(models, name):
    """`LocalModel.generate`: the scheduler admits, cuts prompts into portions, decodes through captured graphs and
    gives slots to later requests; the tokens are the plain implementation's greedy ones."""
    from cuca_b200 import BatchingConfig, LocalModel, LocalModelConfig
    folder, cfg, oracle = models[name]
    prompts = [bu.random_tokens(n, cfg["vocab"], seed=40 + n) for n in (3, 50, 21, 9, 70)]
    model = LocalModel.load(LocalModelConfig(source=str(folder), dtype="float32", context_length=256,
                                             batching=BatchingConfig(max_sequences=2, prefill_chunk=16)))
    outs = model.generate(prompts, max_tokens=12, temperature=0.0)
    for prompt, out in zip(prompts, outs):
        assert out.tokens == _plain_greedy(cfg, oracle.w, prompt, 12)
    stats = model.serving_stats()
    assert stats is not None


def test_command_line_sampling_and_the_prefix_cache_refusal(models):
    """`python -m cuca_b200` on a Bananex folder; seeded sampling is repeatable and differs from greedy somewhere;
    the prefix cache is refused (the layers keep state that cached pages do not bring back)."""
    import subprocess
    import sys
    from pathlib import Path

    from cuca_b200 import BatchingConfig, LocalModel, LocalModelConfig
    from cuca_b200.cache.pages import StatefulCacheError
    folder, cfg, oracle = models["once"]
    root = Path(__file__).resolve().parent.parent
    r = subprocess.run([sys.executable, "-m", "cuca_b200", "--model-dir", str(folder), "--prompt", "5 9 20 31",
                        "--max-tokens", "6", "--temperature", "0", "--dtype", "float32"],
                       capture_output=True, text=True, cwd=root, timeout=600)
    assert r.returncode == 0, r.stderr[-2000:]
    assert [int(t) for t in r.stdout.split()] == _plain_greedy(cfg, oracle.w, [5, 9, 20, 31], 6)
    model = LocalModel.load(LocalModelConfig(source=str(folder), dtype="bfloat16", context_length=128))
    prompt = bu.random_tokens(20, cfg["vocab"], 77)
    a = model.generate(prompt, max_tokens=16, temperature=1.0, top_k=20, seed=5).tokens
    b = model.generate(prompt, max_tokens=16, temperature=1.0, top_k=20, seed=5).tokens
    c = model.generate(prompt, max_tokens=16, temperature=1.0, top_k=20, seed=6).tokens
    assert a == b and a != c and all(0 <= t < cfg["vocab"] for t in a)
    with pytest.raises(StatefulCacheError):
        LocalModel.load(LocalModelConfig(source=str(folder), dtype="bfloat16", context_length=128,
                                         batching=BatchingConfig(prefix_cache=True)))


def test_bfloat16_generation_through_captured_graphs(models):
    """The serving precision end to end: prompts in portions, decode steps replayed as CUDA graphs (the tensor-core
    attention's single-token form with its key tiles dealt to several CTAs, the few-row contractions). Where two
    logits nearly tie bfloat16 may take the other branch, so every token it takes must be a near-maximum of the
    plain implementation's logits at its place."""
    from cuca_b200 import BatchingConfig, LocalModel, LocalModelConfig
    folder, cfg, oracle = models["wide"]
    prompts = [bu.random_tokens(n, cfg["vocab"], seed=60 + n) for n in (5, 70, 33)]
    model = LocalModel.load(LocalModelConfig(source=str(folder), dtype="bfloat16", context_length=256,
                                             batching=BatchingConfig(max_sequences=4, prefill_chunk=32)))
    assert model.backend.use_graphs
    outs = model.generate(prompts, max_tokens=40, temperature=0.0)
    assert model.backend.graph_steps > 0
    for prompt, out in zip(prompts, outs):
        ref = pb.forward(cfg, oracle.w, prompt + out.tokens)
        for i, tok in enumerate(out.tokens):
            row = ref[len(prompt) - 1 + i]
            assert float(row.max() - row[tok]) < 0.05 * float(np.abs(row).max()), (i, tok, int(row.argmax()))
