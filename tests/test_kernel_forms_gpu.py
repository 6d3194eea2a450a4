"""Forms of the kernels that only some sizes reach: each against the kernels it stands in for, or a 64-bit restatement."""
import numpy as np
import pytest
import torch

import plain_model as plain
from test_kernels_gpu import close, data, ops, paged_setup

pytestmark = pytest.mark.gpu

DEV = "cuda:0"
BF = torch.bfloat16


@pytest.mark.parametrize("H,KV,dh", [(36, 2, 64), (16, 2, 128), (33, 3, 64), (17, 1, 128)])
def test_qkv_rope_in_tiles_of_256_columns(H, KV, dh):
    """2,001 rows of about 2,500 columns run in 256-wide tiles, whose epilogue takes two items of a head a warp (the last
    tile of 33 + 6 or 17 + 2 heads overhangs the columns): q, keys and values against the kernels it replaces."""
    o = ops()
    page, d = 16, 72
    ctx_lens, q_lens = [1400, 900, 301], [1000, 700, 301]
    s = paged_setup(ctx_lens, q_lens, KV, dh, page, BF, 9)
    s2 = paged_setup(ctx_lens, q_lens, KV, dh, page, BF, 9)
    T = s["T"]
    x = (data((T, d), 41) * 0.5).to(BF)
    w = (data(((H + 2 * KV) * dh, d), 43) * 0.2).to(BF)
    b = (data(((H + 2 * KV) * dh,), 44) * 0.5).to(BF)
    j = np.arange(dh // 2, dtype=np.float32)
    inv = torch.from_numpy(np.float32(1.0) / np.power(np.float32(1.0e4), (np.float32(2.0) * j) / np.float32(dh), dtype=np.float32)).to(DEV)
    qkv = torch.empty(T, (H + 2 * KV) * dh, device=DEV)
    o.gemm_plain(x, w, qkv, b, o.EPI_BIAS)
    q_ref = torch.empty(T, H * dh, dtype=BF, device=DEV)
    o.rope_kv_write(qkv, s["positions"], s["tok_req"], s["table"], inv, dh // 2, 1.0, q_ref, s["kc"], s["vc"], H, KV, dh, 0)
    cs, sn = o.rope_table(s2["positions"], inv, dh // 2, 1.0)
    q = torch.full((T, H * dh), float("nan"), dtype=BF, device=DEV)
    o.qkv_rope_tc(x, w, b, s2["positions"], s2["tok_req"], s2["table"], cs, sn, q, s2["kc"], s2["vc"], H, KV, dh)
    o.check_status()
    close(q, q_ref.double(), BF, "q")
    pos, req = torch.from_numpy(s["positions_np"]).long(), torch.from_numpy(s["tok_req_np"]).long()
    pages = torch.from_numpy(s["table_np"]).long()[req, pos // page].to(DEV)
    rows = (pos % page).to(DEV)
    for name in ("kc", "vc"):
        close(s2[name][pages, :, rows], s[name][pages, :, rows].double(), BF, name)


@pytest.mark.parametrize("M,N", [(2001, 2048), (1793, 2052), (2304, 2304)])
def test_residual_norm_in_tiles_of_256_columns(M, N):
    """One round of 256-wide tiles where 128-wide ones would take two: the stream, the rows of the pending norm and their
    sums of squares (one part per tile and half)."""
    o = ops()
    K = 72
    x = (data((M, K), 51) * 0.5).to(BF)
    w = (data((N, K), 52) * 0.2).to(BF)
    stream = data((M, N), 53) * 2
    nw = (data((N,), 54) * 0.25 + 1).to(BF)
    want = stream.double().cpu() + x.double().cpu() @ w.double().cpu().T
    out = stream.clone()
    hw, ss = o.gemm_residual_norm(x, w, out, nw)
    o.check_status()
    assert ss.shape[1] == 2 * (-(-N // 256))
    close(out, want, torch.float32, "stream")
    close(hw, want * nw.double().cpu(), BF, "stream times weight")
    close(ss.sum(dim=1), (want * want).sum(dim=1), torch.float32, "sums of squares")


@pytest.mark.parametrize("d", [4, 508, 516, 1024, 1028, 2048, 2052, 4096])
def test_layer_end_chain_at_the_widths_where_its_registers_change(d):
    """The chain of norms at the edges of its forms, against the kernels it stands in for (bit for bit)."""
    o = ops()
    rows, n = 5, 3
    streams = data((n + 1, rows, d), 61) * 2
    sub, gate, gb = data((rows, d), 62), data((rows, d), 63), (data((d,), 64)).to(BF)
    pw, pb, tw, tb = ((data((d,), 65 + i) * 0.25 + 1).to(BF) for i in range(4))
    c = data((n,), 70)
    ref = streams.clone()
    o.gated_norm_residual(ref[n - 1], sub, gate, pw, pb, 1e-6, gb)
    o.depth_mix(ref, c, n, ref[n])
    y_ref = torch.empty(rows, d, dtype=BF, device=DEV)
    o.layernorm(ref[n], tw, tb, 1e-5, y_ref)
    y = torch.empty_like(y_ref)
    o.norm_chain(streams[n - 1], sub, gate, gb, (pw, pb, 1e-6), streams=streams, coeffs=c, n=n, mix_out=streams[n],
                 then=(tw, tb, 1e-5), y=y)
    assert torch.equal(streams, ref) and torch.equal(y, y_ref)


@pytest.mark.parametrize("d", [1020, 1024, 1028, 2048, 2052, 4092, 4096, 4100])
@pytest.mark.parametrize("wdtype", [torch.float32, BF])
def test_rms_norm_at_the_widths_where_its_registers_change(d, wdtype):
    o = ops()
    x = data((7, d), 2) * 3
    w = (data((d,), 3) * 0.25 + 1).to(wdtype)
    for ydtype in (torch.float32, BF):
        y = torch.empty(7, d, dtype=ydtype, device=DEV)
        o.rmsnorm(x, w, 1e-5, y)
        close(y, plain.rms_norm(x.double().cpu(), w.double().cpu(), 1e-5), ydtype, "rmsnorm")


@pytest.mark.parametrize("M,H,KV,dh,d", [(1, 2, 1, 64, 72), (9, 14, 2, 64, 1032), (16, 4, 2, 128, 3584), (17, 6, 2, 32, 520),
                                         (33, 14, 2, 64, 896), (64, 2, 2, 16, 2056)])
@pytest.mark.parametrize("layout", [0, 1])
def test_qkv_rope_of_rows_that_are_normed_already(M, H, KV, dh, d, layout):
    """The q/k/v product of a decode step that reads normed rows, at the edges of its row groups and with K that is no multiple of
    its batches, against the kernels it replaces (product with bias, rotation and cache write)."""
    o = ops()
    page = 16
    ctx_lens, q_lens = [3 + 5 * (i % 40) for i in range(M)], [1] * M
    s = paged_setup(ctx_lens, q_lens, KV, dh, page, BF, 9)
    s2 = paged_setup(ctx_lens, q_lens, KV, dh, page, BF, 9)
    x = data((M, d), 41) * 2
    nw = (data((d,), 42) * 0.25 + 1).to(BF)
    w = (data(((H + 2 * KV) * dh, d), 43) * 0.2).to(BF)
    b = (data(((H + 2 * KV) * dh,), 44) * 0.5).to(BF)
    inv = torch.from_numpy(np.float32(1.0e4) ** (-np.arange(dh // 2, dtype=np.float32) * 2 / dh)).to(DEV)
    h = torch.empty(M, d, dtype=BF, device=DEV)
    o.rmsnorm(x, nw, 1e-6, h)
    qkv = torch.empty(M, (H + 2 * KV) * dh, device=DEV)
    o.gemm_plain(h, w, qkv, b, o.EPI_BIAS)
    q_ref = torch.empty(M, H * dh, dtype=BF, device=DEV)
    o.rope_kv_write(qkv, s["positions"], s["tok_req"], s["table"], inv, dh // 2, 1.0, q_ref, s["kc"], s["vc"], H, KV, dh, layout)
    q = torch.full((M, H * dh), float("nan"), dtype=BF, device=DEV)
    inside = o.norm_inside_qkv
    o.norm_inside_qkv = lambda M, K: False
    try:
        o.norm_qkv_rope(x, nw, 1e-6, w, b, s2["positions"], s2["tok_req"], s2["table"], inv, 1.0, q, s2["kc"], s2["vc"], H, KV, dh, layout)
    finally:
        o.norm_inside_qkv = inside
    close(q, q_ref.double(), BF, "q")
    pos, req = torch.from_numpy(s["positions_np"]).long(), torch.from_numpy(s["tok_req_np"]).long()
    pages = torch.from_numpy(s["table_np"]).long()[req, pos // page].to(DEV)
    rows = (pos % page).to(DEV)
    for name in ("kc", "vc"):
        close(s2[name][pages, :, rows], s[name][pages, :, rows].double(), BF, name)


def _scan64(rule, q, k, v, a, b, scale, S, H):
    """The recurrence of one request in 64 bits: rows q, k, a [n, H, dk], v [n, H, dv], b [n, H]; S [H, dk, dv] is left updated."""
    o = ops()
    out = torch.zeros_like(v)
    for t in range(q.shape[0]):
        if rule == o.RULE_BONUS:
            out[t] = (torch.einsum("hkv,hk->hv", S, q[t]) + b[t][:, None] * v[t]) * scale
        S *= a[t][:, :, None]
        u = v[t] if rule != o.RULE_DELTA else torch.sigmoid(b[t])[:, None] * (v[t] - torch.einsum("hkv,hk->hv", S, k[t]))
        S += k[t][:, :, None] * u[:, None]
        if rule != o.RULE_BONUS:
            out[t] = torch.einsum("hkv,hk->hv", S, q[t]) * scale
    return out


@pytest.mark.parametrize("rule", ["RULE_GLA", "RULE_DELTA", "RULE_BONUS"])
@pytest.mark.parametrize("H,dk,dv,lens", [(2, 64, 128, [257, 5, 0, 700]), (3, 128, 40, [256, 255]), (1, 16, 33, [300]), (5, 32, 256, [1, 512, 3, 9, 1, 1])])
@pytest.mark.parametrize("parts", [1, 2, 9, 32, 300])
def test_scan_in_parts(rule, H, dk, dv, lens, parts):
    """Portions cut into parts (more parts than tokens among them) beside short ones and requests without tokens, few blocks and
    many (the two forms of the kernel): outputs and states against 64 bits, and slots that no request owns stay as they are."""
    o = ops()
    rule = getattr(o, rule)
    T, R = sum(lens), len(lens)
    g = torch.Generator().manual_seed(T + parts)
    rnd = lambda *n: torch.randn(*n, generator=g)
    q, k, v, b = rnd(T, H * dk) * 0.3, rnd(T, H * dk), rnd(T, H * dv), rnd(T, H)
    k = (k.view(T, H, dk) / k.view(T, H, dk).norm(dim=-1, keepdim=True)).reshape(T, H * dk)
    a = torch.sigmoid(rnd(T, H * dk) + 3.0)
    state = rnd(R + 2, H * dk * dv)
    slots = torch.arange(R, 0, -1, dtype=torch.int32)
    cu = torch.tensor([0] + lens, dtype=torch.int32).cumsum(0).to(torch.int32)
    dev = lambda t: t.to(DEV)
    st = dev(state.clone())
    out = torch.full((T, H * dv), float("nan"), device=DEV)
    o.recurrent_scan(rule, dev(q), dev(k), dev(v), dev(a), None if rule == o.RULE_GLA else dev(b), 0.5, st, dev(slots), dev(cu), out,
                     H, H, dk, dv, parts=parts)
    want_state = state.double().clone()
    for r in range(R):
        lo, hi = int(cu[r]), int(cu[r + 1])
        if hi == lo:
            continue
        S = want_state[int(slots[r])].view(H, dk, dv)
        w = _scan64(rule, *(x[lo:hi].double().view(hi - lo, H, -1) for x in (q, k, v, a)), b[lo:hi].double(), 0.5, S, H)
        close(out[lo:hi], w.reshape(hi - lo, -1), torch.float32, f"outputs of request {r}")
    close(st, want_state, torch.float32, "states")
    assert torch.equal(st[0].cpu(), state[0]) and torch.equal(st[R + 1].cpu(), state[R + 1])


@pytest.mark.parametrize("rule", ["RULE_GLA", "RULE_DELTA", "RULE_BONUS"])
@pytest.mark.parametrize("lens,n_long", [([3, 300, 1, 0, 257, 1], 2), ([1] * 130 + [256, 1, 400], 2), ([300, 270, 1, 290], 1), ([1, 260], 0)])
def test_scan_keeps_scratch_for_the_requests_that_are_cut(rule, lens, n_long):
    """Long portions among short ones: scratch by long request and not by request; long portions past the number given (the last
    two cases) are walked in one piece. Outputs and states against 64 bits."""
    o = ops()
    rule = getattr(o, rule)
    H, dk, dv, parts = 2, 32, 40, 6
    T, R = sum(lens), len(lens)
    g = torch.Generator().manual_seed(T)
    rnd = lambda *n: torch.randn(*n, generator=g)
    q, k, v, b = rnd(T, H * dk) * 0.3, rnd(T, H * dk), rnd(T, H * dv), rnd(T, H)
    k = (k.view(T, H, dk) / k.view(T, H, dk).norm(dim=-1, keepdim=True)).reshape(T, H * dk)
    a = torch.sigmoid(rnd(T, H * dk) + 3.0)
    state = rnd(R, H * dk * dv)
    cu = torch.tensor([0] + lens, dtype=torch.int32).cumsum(0).to(torch.int32)
    args = [t.to(DEV) for t in (q, k, v, a)] + [None if rule == o.RULE_GLA else b.to(DEV), 0.5]
    st, out = state.to(DEV), torch.full((T, H * dv), float("nan"), device=DEV)
    slots, cud = torch.arange(R, dtype=torch.int32, device=DEV), cu.to(DEV)
    torch.cuda.synchronize()
    torch.cuda.reset_peak_memory_stats()
    before = torch.cuda.memory_allocated()
    o.recurrent_scan(rule, *args, st, slots, cud, out, H, H, dk, dv, parts=parts, n_long=n_long)
    per = dk * (2 * dv + dk) if rule == o.RULE_DELTA else dk * (dv + 1)
    assert torch.cuda.max_memory_allocated() - before <= n_long * parts * H * per * 4 + 4 * R + 1024
    want_state = state.double()
    for r in range(R):
        lo, hi = int(cu[r]), int(cu[r + 1])
        if hi > lo:
            w = _scan64(rule, *(x[lo:hi].double().view(hi - lo, H, -1) for x in (q, k, v, a)), b[lo:hi].double(), 0.5,
                        want_state[r].view(H, dk, dv), H)
            close(out[lo:hi], w.reshape(hi - lo, -1), torch.float32, f"outputs of request {r}")
    close(st, want_state, torch.float32, "states")


@pytest.mark.parametrize("rule", ["RULE_GLA", "RULE_DELTA", "RULE_BONUS"])
def test_scan_takes_blocks_by_the_portions_under_way(rule):
    """The requests of a few tokens beside a long portion are not counted as if they kept the launch busy, and both builds
    of the kernel give the same bits."""
    from boring_llm_b200.parts.recurrent import GatedLinearAttention
    o = ops()
    rule = getattr(o, rule)
    H, dk, dv, lens = 4, 64, 256, [200] + [1] * 40
    mixer = GatedLinearAttention(64, H, dk, dv, 16.0, 1e-6, {})
    assert [mixer._cut(x)["busy"] for x in ([2000] + [1] * 31, [1] * 64, [200, 100] + [50] * 12, [0, 0])] == [1, 64, 4, 1]
    T, R = sum(lens), len(lens)
    q, k, v, b = data((T, H * dk), 1) * 0.3, data((T, H * dk), 2) * 0.1, data((T, H * dv), 3), data((T, H), 4)
    a = torch.sigmoid(data((T, H * dk), 5) + 3.0)
    cu = torch.tensor([0] + lens, device=DEV).cumsum(0).to(torch.int32)
    got = []
    for busy in (1, R, None):
        st, out = data((R, H * dk * dv), 6), torch.full((T, H * dv), float("nan"), device=DEV)
        o.recurrent_scan(rule, q, k, v, a, None if rule == o.RULE_GLA else b, 0.5, st, torch.arange(R, dtype=torch.int32, device=DEV), cu, out,
                         H, H, dk, dv, busy=busy)
        got.append((out, st))
    assert all(torch.equal(x, y) for other in got[1:] for x, y in zip(got[0], other))


def test_scans_are_cut_where_that_was_measured_to_pay():
    """One long portion at two sizes: a cut of linear attention pays at both (few parts at the larger, where every further round
    of blocks costs), of the delta rule only at the smaller, whose fold is short; several long portions fill the device."""
    o = ops()
    parts = o.recurrent_scan_parts
    assert parts(o.RULE_DELTA, 8, 128, 256, 1) == 1
    assert 4 <= parts(o.RULE_GLA, 8, 128, 256, 1) <= 12
    assert 8 <= parts(o.RULE_DELTA, 7, 64, 128, 1) <= 12 and 16 <= parts(o.RULE_GLA, 7, 64, 128, 1) <= 21
    assert 4 <= parts(o.RULE_DELTA, 7, 64, 128, 1, 256) <= 8 and parts(o.RULE_DELTA, 7, 64, 128, 1, 2048) == 14
    assert parts(o.RULE_GLA, 8, 128, 256, 2) == 1 and parts(o.RULE_GLA, 7, 64, 128, 8) == 1 and parts(o.RULE_GLA, 7, 64, 128, 0) == 1


@pytest.mark.parametrize("taps,C,unit,dk", [(4, 96, 4, 16), (4, 2052, 2, 130), (4, 8200, 8, 1024), (3, 96, 4, 16), (4, 90, 4, 16)])
def test_short_convolution_forms(taps, C, unit, dk):
    """Four taps of channels in groups of four, and what does not fit that form, against 64 bits: requests that begin here,
    go on from a slot's tail, have one token or none."""
    o = ops()
    lens = [5, 1, 0, 2, 40]
    T, R = sum(lens), len(lens)
    ld = C + 12
    x, tail = data((T, ld), 3), data((R + 1, (taps - 1) * C + 4), 5)
    w, bias = data((C, taps), 7), data((C,), 8)
    slots = torch.tensor([4, 2, 0, 1, 3], dtype=torch.int32, device=DEV)
    cu = torch.tensor([0] + lens).cumsum(0).to(torch.int32)
    req = torch.repeat_interleave(torch.arange(R), torch.tensor(lens)).to(torch.int32)
    for b in (None, bias):
        y = torch.full((T, C), float("nan"), device=DEV)
        o.conv_silu_unit(x, w, tail, slots, req.to(DEV), cu.to(DEV), y, unit, 1, dk, 0.25, 1e-6, bias=b)
        for r in range(R):
            lo, hi = int(cu[r]), int(cu[r + 1])
            if lo == hi:
                continue
            rows = torch.cat([tail[int(slots[r]), :(taps - 1) * C].view(taps - 1, C), x[lo:hi, :C]]).double().cpu()
            z = sum(rows[i:i + hi - lo] * w[:, i].double().cpu() for i in range(taps)) + (0 if b is None else b.double().cpu())
            z = z * torch.sigmoid(z)
            u = z[:, :unit * dk].reshape(hi - lo, unit, dk)
            u = u / torch.sqrt((u * u).sum(-1, keepdim=True) + 1e-6)
            u[:, 0] *= 0.25
            z[:, :unit * dk] = u.reshape(hi - lo, -1)
            close(y[lo:hi], z, torch.float32, f"request {r}")


@pytest.mark.parametrize("H,N,T,gate_heads", [(3, 20, 5, False), (2, 128, 300, True), (3, 18, 4, False), (1, 4, 1, None)])
def test_gated_head_rows_forms(H, N, T, gate_heads):
    o = ops()
    Tp = T + 3
    hv = data((H, Tp, N), 3)
    gate = None if gate_heads is None else data((T, (H if gate_heads else H * N) + 4), 4)
    out = torch.empty(T, H * N, dtype=BF, device=DEV)
    o.heads_gate_rows(hv, None if gate is None else gate[:, :(H if gate_heads else H * N)], out, gate_heads=bool(gate_heads))
    want = hv[:, :T].double().cpu().permute(1, 0, 2)
    if gate is not None:
        g = torch.sigmoid(gate.double().cpu())
        want = want * (g[:, :H, None] if gate_heads else g[:, :H * N].view(T, H, N))
    close(out, want.reshape(T, H * N), BF, "gated rows")


@pytest.mark.parametrize("d,top", [(4, 1), (36, 3), (2052, 2), (30, 2), (1028, 9)])
@pytest.mark.parametrize("add", [False, True])
def test_combined_expert_rows_forms(d, top, add):
    o = ops()
    T = 7
    y, x = data((T * top + 5, d), 3), data((T, d), 4).to(BF)
    pos = (torch.arange(T * top, dtype=torch.int32) * 3) % (T * top + 5)
    pos[::4] = -1                                             # pairs without a row: the token's own
    wts, out = data((T, top), 6), data((T, d), 7)
    want = out.double().cpu() if add else torch.zeros(T, d, dtype=torch.float64)
    for p in range(T * top):
        row = x[p // top] if pos[p] < 0 else y[int(pos[p])]
        want[p // top] += wts[p // top, p % top].double().cpu() * row.double().cpu()
    o.moe_combine_rows(y, pos.to(DEV), wts, out, add=add, x=x)
    close(out, want, torch.float32, "combined rows")


@pytest.mark.parametrize("M,N,n_act,K", [(256, 8, 4, 64), (300, 200, 200, 72), (700, 1000, 620, 136), (2048, 5760, 4864, 64), (257, 300, 36, 8)])
@pytest.mark.parametrize("act", [0, 1, 2])
def test_activation_in_the_epilogue_of_the_product_on_pairs(M, N, n_act, K, act):
    """The activated columns and the further 32-bit columns behind them equal the product and the activation in launches of their
    own, bit for bit; widths that cut a chunk of 32 columns, tiles of 128 and of 256, no further columns."""
    o = ops()
    x, w = (data((M, K), 1) * 0.5).to(BF), (data((N, K), 2) * 0.3).to(BF)
    sums = torch.empty(M, N, device=DEV)
    o.gemm_tc_pair(x, w, sums)
    want = torch.empty(M, n_act, dtype=BF, device=DEV)
    o.activation(sums[:, :n_act], want, act)
    y = torch.full((M, n_act), float("nan"), dtype=BF, device=DEV)
    assert o.gemm_kernel(x, w, N, None, o.EPI_NONE) == "pair"
    rest = o.linear_act(x, w, y, act)
    o.check_status()
    assert torch.equal(y, want)
    assert (rest is None) == (N == n_act) and (rest is None or torch.equal(rest, sums[:, n_act:]))


@pytest.mark.parametrize("M", [64, 300])
def test_activated_product_over_its_own_rows(M):
    """out in the place of x: no tile is written while another still reads, so the product has a launch of its own."""
    o = ops()
    x, w = (data((M, 1024), 1) * 0.5).to(BF), (data((1024, 1024), 2) * 0.05).to(BF)
    want = torch.empty(M, 1024, dtype=BF, device=DEV)
    seen = []
    call = o._call

    def spy(fn, *a):
        seen.append(fn.__name__)
        return call(fn, *a)
    o._call = spy
    try:
        assert o.linear_act(x, w, want, 1) is None
        assert ("bl_gemm_tc_pair_act" in seen) == (M >= 256)
        seen.clear()
        assert o.linear_act(x, w, x, 1) is None
        assert "bl_gemm_tc_pair_act" not in seen
    finally:
        o._call = call
    o.check_status()
    assert torch.equal(x, want)


@pytest.mark.parametrize("K", [4, 28, 32, 36, 896])
@pytest.mark.parametrize("M,N", [(1, 16), (3, 70), (17, 33), (65, 100), (366, 257)])
def test_32_bit_product_does_not_depend_on_the_rows_beside_a_row(M, N, K):
    """The 32-bit tiles (chosen by the number of rows) at edges of rows, columns and stages, with rows of x that lie further apart
    than they are long: 64 bits, and the same bits for a row alone."""
    o = ops()
    full = data((M, K + 8), 1)
    x, w, b = full[:, :K], data((N, K), 2) * 0.3, data((N,), 3)
    out = torch.empty(M, N, device=DEV)
    xc = x.contiguous()
    o.gemm_plain(xc, w, out, b, o.EPI_BIAS)
    close(out, xc.double().cpu() @ w.double().cpu().T + b.double().cpu(), torch.float32, "product")
    one = torch.empty(1, N, device=DEV)
    o.gemm_plain(xc[M // 2:M // 2 + 1], w, one, b, o.EPI_BIAS)
    assert torch.equal(one[0], out[M // 2])
    strided = torch.empty(M, N, device=DEV)
    o.gemm_plain(x, w, strided, b, o.EPI_BIAS)
    assert torch.equal(strided, out)


@pytest.mark.parametrize("M,N,K,kind", [(8, 256, 8192, "skinny"), (9, 256, 8192, "splitk"), (16, 200, 8200, "splitk"), (16, 256, 8184, "skinny"),
                                        (17, 136, 4096, "splitk"), (31, 1024, 4104, "splitk"), (16, 256, 4096, "skinny"),
                                        (32, 9473, 72, "cols"), (1, 9480, 520, "cols"), (8, 9472, 72, "skinny")])
def test_products_of_few_rows_at_the_lines_between_their_kernels(M, N, K, kind):
    """The kernel that the dispatch takes on either side of a line, and its result against 64 bits."""
    o = ops()
    x, w = (data((M, K), 1) * 0.5).to(BF), (data((N, K), 2) * 0.2).to(BF)
    epi = o.EPI_NONE if kind == "cols" or N == 9472 else o.EPI_RESIDUAL
    out = data((M, N), 3)
    want = x.double().cpu() @ w.double().cpu().T + (out.double().cpu() if epi == o.EPI_RESIDUAL else 0.0)
    assert o.gemm_kernel(x, w, N, None, epi) == kind
    o.gemm(x, w, out, None, epi)
    o.check_status()
    close(out, want, BF, "product")


@pytest.mark.parametrize("M,N,K", [(256, 256, 64), (300, 19000, 72), (513, 40000, 136), (2048, 896, 896)])
def test_products_on_pairs_one_behind_the_other(M, N, K):
    """One to five tiles a pair, launch upon launch (the next one's blocks move in as the last one's leave): the same bits
    every time, and those are the product's."""
    o = ops()
    x, w = (data((M, K), 1) * 0.5).to(BF), (data((N, K), 2) * 0.2).to(BF)
    outs = [torch.full((M, N), float("nan"), device=DEV) for _ in range(4)]
    for i in range(40):
        o.gemm_tc_pair(x, w, outs[i % 4])
        if i % 4 == 3:
            assert all(torch.equal(outs[0], t) for t in outs[1:])
    o.check_status()
    want = torch.empty(M, N, device=DEV)
    o.gemm_plain(x, w, want)
    close(outs[0], want.double(), torch.float32, "product")


@pytest.mark.parametrize("rank,rot", [(8, 8), (128, 32), (136, 8), (504, 16), (512, 64)])
@pytest.mark.parametrize("window,contexts", [(0, [1100, 70, 1]), (130, [1100, 129, 40])])
def test_slices_of_a_token_with_a_long_context(rank, rot, window, contexts):
    """A token's keys in 15, 16 and 17 slices (the merge holds up to 16 in a thread's registers, 128 columns at a time) and in more
    slices than there are key blocks: slices without keys leave their sums of earlier memory, which is NaN here, alone."""
    import plain_miforax as pm
    o = ops()
    if not o.latent_attention_mma_supported(BF, rank, rot, 16):
        pytest.skip("sizes that the kernel does not take")
    H, R, dk, scale = 3, len(contexts), rank + rot, 0.3
    g = torch.Generator().manual_seed(rank + window)
    rows = [(torch.randn(n, dk, generator=g, dtype=torch.float64) * 0.5).to(BF).double() for n in contexts]
    q = (torch.randn(R, H, dk, generator=g, dtype=torch.float64) * 0.5).to(BF).double()
    sinks = torch.randn(H, generator=g, dtype=torch.float64)
    width = -(-max(contexts) // 16)
    cache = torch.full((R * width, 1, 16, dk), float("nan"), dtype=BF)
    table = torch.arange(R * width, dtype=torch.int32).flip(0).reshape(R, width)
    want = torch.empty(H, R, rank, dtype=torch.float64)
    for r, n in enumerate(contexts):
        for j in range(n):
            cache[table[r, j // 16], 0, j % 16] = rows[r][j].to(BF)
        k = rows[r][None].expand(H, n, dk)
        seen = torch.arange(n) >= (n - window if window else 0)
        want[:, r] = pm.sink_softmax_attention(q[r][:, None], k, k[:, :, :rank], scale, sinks, seen[None])[:, 0]
    i32 = lambda t: torch.tensor(t, dtype=torch.int32, device=DEV)
    head_major = lambda t: t.permute(1, 0, 2).to(BF).contiguous().to(DEV)
    args = (head_major(q[:, :, :rank]), head_major(q[:, :, rank:]), cache.to(DEV), i32(list(range(R + 1))), i32(contexts), table.to(DEV), i32(list(range(R))))
    for splits in (1, 15, 16, 17, 40):
        poison = torch.full((4, H * R * splits * max(rank, 2)), float("nan"), device=DEV)
        torch.cuda.synchronize()
        del poison                                            # what the scratch is taken from
        out = torch.full((H, R, rank), float("nan"), dtype=BF, device=DEV)
        o.latent_attention_mma(*args, True, out, window, scale, sinks.float().to(DEV), splits)
        assert torch.isfinite(out).all()
        close(out, want, BF, f"{splits} slices")              # (weights and results of 8 bits, as the kernels' other tests take them)


@pytest.mark.parametrize("q_rank,rank,rot_dim,dims", [(127, 129, 8, 8), (128, 128, 16, 12), (1024, 1024, 64, 64), (1025, 40, 8, 8), (40, 1025, 8, 4),
                                                      (129, 520, 128, 128), (24, 16, 130, 130)])
@pytest.mark.parametrize("dtype", [torch.float32, BF])
def test_latent_rows_at_the_widths_where_their_form_changes(q_rank, rank, rot_dim, dims, dtype):
    """Both norms, the rotation and the cache row with all values in registers (up to 1,024 a norm, 128 of the shared key part) and
    read in loops; either result left out. NaN in what a form must not read."""
    o = ops()
    T, eps, mscale = 5, 1e-5, 1.25
    positions = [37, 5, 16, 0, 31]
    proj = data((T, q_rank + rank + rot_dim + 9), 1)
    off_q, off_kv = 3, q_rank + 5
    qw, kw = (data((q_rank,), 2) * 0.25 + 1).to(dtype), (data((rank,), 3) * 0.25 + 1).to(dtype)
    inv = torch.tensor([100.0 ** (-2.0 * j / dims) for j in range(dims // 2)], device=DEV)
    i32 = lambda t: torch.tensor(t, dtype=torch.int32, device=DEV)
    table = i32([[4, 7, 2], [6, 1, 0], [3, 5, 8]])
    req = [0, 1, 2, 2, 1]
    p = proj.double().cpu()
    zq, zk, zr = p[:, off_q:off_q + q_rank], p[:, off_kv:off_kv + rank], p[:, off_kv + rank:off_kv + rank + rot_dim]
    a = torch.tensor(positions, dtype=torch.float64)[:, None] * inv.double().cpu()
    u, v, h = zr[:, :dims // 2], zr[:, dims // 2:dims], zr[:, dims:]
    turned = torch.cat([(u * a.cos() - v * a.sin()) * mscale, (v * a.cos() + u * a.sin()) * mscale, h], 1)
    want_q = plain.rms_norm(zq, qw.double().cpu(), eps)
    want_row = torch.cat([plain.rms_norm(zk, kw.double().cpu(), eps), turned], 1)
    for with_q, with_row in ((True, True), (True, False), (False, True)):
        x = proj.clone()
        if not with_q:
            x[:, off_q:off_q + q_rank] = float("nan")
        if not with_row:
            x[:, off_kv:] = float("nan")
        cq = torch.full((T, q_rank), float("nan"), dtype=dtype, device=DEV) if with_q else None
        cache = torch.full((9, 1, 16, rank + rot_dim), float("nan"), dtype=dtype, device=DEV) if with_row else None
        o.latent_prep(x, off_q, q_rank, off_kv, rank, rot_dim, dims // 2, qw if with_q else None, kw if with_row else None, eps,
                      i32(positions), i32(req), table, inv, mscale, cq, cache)
        if with_q:
            close(cq, want_q, dtype, "query latent")
        if with_row:
            at = [(int(table[r, t // 16]), t % 16) for r, t in zip(req, positions)]
            close(torch.stack([cache[pg, 0, s] for pg, s in at]), want_row, dtype, "cache rows")
            assert int(torch.isfinite(cache).all(-1).sum()) == T


@pytest.mark.parametrize("T,H", [(1, 3), (256, 9), (257, 9), (256, 8), (300, 2), (2, 17)])
@pytest.mark.parametrize("n,rot_half,n_lead,gap", [(32, 16, 64, 0), (32, 12, 62, 2), (8, 4, 4, 1), (10, 5, 0, 0), (64, 32, 128, 4)])
@pytest.mark.parametrize("dtype", [torch.float32, BF])
def test_turned_heads_in_shares(T, H, n, rot_half, n_lead, gap, dtype):
    """Up to 256 tokens a token's heads lie on several blocks, of unequal shares where eight do not divide them; the other slice in
    16-byte pieces where sizes and strides allow, else value by value."""
    o = ops()
    width = n_lead + n + gap
    x = data((T, H * width), 1).view(T, H, width)
    lead, q = (x[:, :, :n_lead] if n_lead else None), x[:, :, n_lead:n_lead + n]
    positions = torch.arange(T, dtype=torch.int32, device=DEV) * 3 % 97
    inv = torch.tensor([50.0 ** (-j / rot_half) for j in range(rot_half)], device=DEV)
    out = torch.full((T, H, n), float("nan"), dtype=dtype, device=DEV)
    lead_out = torch.full((T, H, n_lead), float("nan"), dtype=dtype, device=DEV) if n_lead else None
    o.rope_heads(q, positions, inv, rot_half, 0.75, out, lead, lead_out)
    a = (positions.double().cpu()[:, None] * inv.double().cpu())[:, None]
    c, s, z = a.cos() * 0.75, a.sin() * 0.75, q.double().cpu()
    u, v = z[:, :, :rot_half], z[:, :, rot_half:2 * rot_half]
    close(out, torch.cat([u * c - v * s, v * c + u * s, z[:, :, 2 * rot_half:]], 2), dtype, "turned heads")
    if n_lead:
        assert torch.equal(lead_out, lead.to(dtype))


@pytest.mark.parametrize("H,own,rot,dv,rank", [(3, 128, 64, 128, 512), (2, 64, 32, 64, 72)])
@pytest.mark.parametrize("window,gate_dim", [(0, 0), (200, 1), (128, 0), (37, 1)])
def test_attention_over_keys_made_of_latents(H, own, rot, dv, rank, window, gate_dim):
    """Portions that end at edges of tiles, key blocks and pages, beside single tokens of short contexts and a request without
    tokens, pages that the window has given back missing from the table and full of NaN: the rows that are copied, bit for bit, and the
    attention against 64 bits on the same bfloat16 operands."""
    from boring_llm_b200.parts.latent import latent_keys_plan
    o = ops()
    ctx = [1, 130, 128, 700, 129, 16, 385, 128, 1]
    q_lens = [1, 130, 127, 300, 1 if window == 0 else 2, 16, 129, 1, 0]
    if window == 0:
        ctx[4], q_lens[4] = 128, 1
    R, T = len(ctx), sum(q_lens)
    plan = latent_keys_plan(q_lens, ctx, R - 1, window, (H, own, rot, dv, 10 ** 6))
    assert plan is not None and plan.shape == ("keys", len(plan.arrays["work"]), R, len(plan.arrays["tiles"]))
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    cu = [0]
    for n in q_lens:
        cu.append(cu[-1] + n)
    dk = rank + rot
    pages = sum(-(-c // 16) for c in ctx) + 1
    cache = data((pages, 1, 16, dk), 1).to(BF)
    width = max(-(-c // 16) for c in ctx) + 2
    table, at, rows = np.full((R, width), -1, np.int32), 1, []
    for r, (c, n) in enumerate(zip(ctx, q_lens)):
        k = -(-c // 16)
        first = max(0, c - max(n, 1) - window + 1) // 16 if window else 0           # the first page that a new token sees
        got = cache[at:at + k, 0].reshape(-1, dk)[:c].clone()
        got[:16 * first] = 0
        cache[at:at + first] = float("nan")
        table[r, first:k] = np.arange(at + first, at + k)
        if c % 16:
            cache[at + k - 1, 0, c % 16:] = float("nan")                            # what an earlier request left behind the last key
        at += k
        rows.append(got)
    L = 16 * len(plan.arrays["work"])
    latent, shared = torch.full((L, rank), 7.0, dtype=BF, device=DEV), torch.full((L, 64), 7.0, dtype=BF, device=DEV)
    o.latent_rows(cache, i32(plan.arrays["work"]), i32(cu), i32(ctx), i32(table), latent, shared)
    key_row = plan.arrays["key_row"]
    starts = [max(0, c - n - window + 1) // 128 * 128 if window else 0 for c, n in zip(ctx, q_lens)]
    for r, (c, n) in enumerate(zip(ctx, q_lens)):
        if n:
            to = int(key_row[r]) + starts[r]
            assert torch.equal(latent[to:to + c - starts[r]], rows[r][starts[r]:, :rank])
            assert torch.equal(shared[to:to + c - starts[r], :rot], rows[r][starts[r]:, rank:])
    assert torch.isfinite(latent.float()).all()
    kv = torch.empty(L, H * (own + dv), dtype=BF, device=DEV)
    o.gemm(latent, (data((H * (own + dv), rank), 2) * rank ** -0.5).to(BF), kv)
    q = data((T, H * (own + rot)), 3).to(BF)
    sinks, gate = data((H,), 4), data((T, H * dv + 4), 5)
    scale = 0.3
    out = torch.full((T, H * dv), float("nan"), dtype=BF, device=DEV)
    o.attention_rows_tc(q, kv, shared, i32(key_row), i32(cu), i32(ctx), i32(plan.arrays["tiles"]), out, H, own, dv, window, scale, sinks,
                        gate if gate_dim else gate[:, :H], gate_dim=dv if gate_dim else 0)
    o.check_status()
    kv64, sh64, q64 = kv.double(), shared.double()[:, :rot], q.double().view(T, H, own + rot)
    for r, (c, n) in enumerate(zip(ctx, q_lens)):
        if not n:
            continue
        span = slice(int(key_row[r]) + starts[r], int(key_row[r]) + c)
        i = torch.arange(c - n, c, device=DEV)[:, None]
        j = torch.arange(starts[r], c, device=DEV)[None, :]
        seen = (j <= i) & ((i - j < window) if window else (j >= 0))
        for h in range(H):
            k = torch.cat([kv64[span, h * own:(h + 1) * own], sh64[span]], dim=1)
            v = kv64[span, H * own + h * dv:H * own + (h + 1) * dv]
            t = slice(cu[r], cu[r + 1])
            s = (q64[t, h] @ k.T * scale).masked_fill(~seen, float("-inf"))
            s = torch.cat([s, sinks[h].double().expand(n, 1)], dim=1)
            want = torch.softmax(s, dim=1)[:, :-1] @ v
            want = want * torch.sigmoid(gate[t, h * dv:(h + 1) * dv].double() if gate_dim else gate[t, h:h + 1].double())
            close(out[t, h * dv:(h + 1) * dv], want, BF, f"request {r} head {h}")


@pytest.mark.parametrize("N,K", [(128, 256), (130, 260), (896, 896), (1152, 900), (4160, 512), (896, 4864), (32772, 256)])
@pytest.mark.parametrize("M", [1, 16, 33, 97, 366])
def test_32_bit_product_on_tensor_cores(M, N, K):
    """Spans of K and none, widths of 16 to 128 rows, remainders of rows, columns and segments, every epilogue: no further from 64
    bits than a chain of FMAs in 32 bits comes (numbers of one sign, where cut-off bits would add up, among them), and the same bits
    for a row alone."""
    o = ops()
    g = torch.Generator().manual_seed(M * 7919 + N + K)
    rnd = lambda *s: torch.randn(*s, generator=g).to(DEV)
    full, w, w2, b = rnd(M, K + 4), rnd(N, K) * 0.3, rnd(2 * N, K) * 0.3, rnd(N)
    x = full[:, :K]

    def rel(got, want):
        return ((got.double() - want).norm() / want.norm()).item()

    out = torch.empty(M, N, device=DEV)
    for x_, w_ in ((x, w), (full.abs()[:, :K], w.abs())):
        o.gemm(x_, w_, out)
        want = x_.double() @ w_.double().T
        assert rel(out, want) <= rel(fma_chain(x_, w_), want)
        close(out, want, torch.float32, "product")
    one = torch.empty(1, N, device=DEV)
    o.gemm(x, w, out, b, o.EPI_BIAS)
    o.gemm(x[M // 2:M // 2 + 1].contiguous(), w, one, b, o.EPI_BIAS)
    assert torch.equal(one[0], out[M // 2])
    res = rnd(M, N)
    want = res.double() + x.double() @ w.double().T
    o.gemm(x, w, res, None, o.EPI_RESIDUAL)
    close(res, want, torch.float32, "residual")
    o.gemm(x, w2, out, None, o.EPI_SWIGLU)
    gu = x.double() @ w2.double().T
    close(out, plain.silu(gu[:, :N]) * gu[:, N:], torch.float32, "swiglu")
    one = torch.empty(1, N, device=DEV)
    o.gemm(x[M - 1:], w2, one, None, o.EPI_SWIGLU)
    assert torch.equal(one[0], out[M - 1])
    o.check_status()


def test_32_bit_product_on_tensor_cores_of_infinities_and_extremes():
    """Rows with an infinity, a NaN, the largest numbers and small ones: what a chain of FMAs gives, and other rows untouched."""
    o = ops()
    g = torch.Generator().manual_seed(5)
    M, N, K = 70, 256, 512
    x, w = torch.randn(M, K, generator=g).to(DEV), torch.randn(N, K, generator=g).to(DEV)
    plainly = torch.empty(M, N, device=DEV)
    o.gemm(x, w, plainly)
    y = x.clone()
    y[3, 7], y[5, 9], y[8, 0], y[11, 500] = float("inf"), float("nan"), -float("inf"), 3.4028234e38
    y[20] *= 1e-30
    y[21] *= 1e30
    v = w.clone()
    v[40, 7] = 0.0                                     # infinity times zero
    v[41] = w[41].bfloat16().float()                   # numbers whose second half is zero
    out = torch.empty(M, N, device=DEV)
    o.gemm(y, v, out)
    want = (y.double() @ v.double().T)
    for r in (3, 8):
        torch.testing.assert_close(out[r].double(), want[r], rtol=0, atol=0, equal_nan=True)
    assert out[5].isnan().all()
    fits = torch.isfinite(want[11].float())
    assert 0 < fits.sum() < N and torch.equal(torch.isfinite(out[11]), fits)
    for r, n in ((11, fits), (20, slice(None)), (21, slice(None))):
        assert ((out[r][n].double() - want[r][n]).norm() / want[r][n].norm()) < 1e-6
    keep = [r for r in range(M) if r not in (3, 5, 8, 11, 20, 21)]
    cols = [n for n in range(N) if n not in (40, 41)]
    assert torch.equal(out[keep][:, cols], plainly[keep][:, cols])
    o.check_status()


def fma_chain(x, w):
    """fmaf in ascending k: the 48-bit product is exact in 64 bits, the sum rounded to 32."""
    acc = torch.zeros(x.shape[0], w.shape[0], device=x.device)
    for k in range(x.shape[1]):
        acc = (acc.double() + x[:, k:k + 1].double() * w[:, k].double()).float()
    return acc


@pytest.mark.parametrize("M,N,K", [(1, 128, 256), (33, 896, 896), (200, 132, 512)])
def test_32_bit_product_without_tensor_cores(M, N, K):
    """`fast=False` and `gemm_plain` are the chain of FMAs, bit for bit, at sizes that the tensor cores take, too; those give other bits."""
    o = ops()
    g = torch.Generator().manual_seed(M + N + K)
    x, w = torch.randn(M, K, generator=g).to(DEV), torch.randn(N, K, generator=g).to(DEV)
    want = fma_chain(x, w)
    out = torch.empty(M, N, device=DEV)
    assert o.gemm_f32_tc_supported(x, w, out)
    o.gemm(x, w, out, fast=False)
    assert torch.equal(out, want)
    out.zero_()
    o.gemm_plain(x, w, out)
    assert torch.equal(out, want)
    o.gemm(x, w, out)
    assert not torch.equal(out, want)
    close(out, x.double() @ w.double().T, torch.float32, "product")
    o.check_status()


@pytest.mark.parametrize("fast", [True, False])
def test_32_bit_steps_with_and_without_tensor_cores(fast, tmp_path):
    """A float32 model at sizes that the tensor cores take: both ways against the plain implementation, and only the fast one asks for
    the status words."""
    import boring_llm_b200 as b
    cfg = b.Qwen2Config.from_dict(dict(
        architectures=["Qwen2ForCausalLM"], num_hidden_layers=2, hidden_size=256, num_attention_heads=4, num_key_value_heads=2,
        intermediate_size=384, vocab_size=300, rope_theta=10000.0, rms_norm_eps=1e-6, tie_word_embeddings=True, max_position_embeddings=128))
    b.write_random_model(str(tmp_path), cfg, 3, "float32", 0.05)
    eng = b.Engine(str(tmp_path), dtype="float32", ctx_size=96, max_num_seqs=2, max_tokens=192)
    eng.runner.fast = fast
    toks = np.random.default_rng(0).integers(0, 300, 70).tolist()
    got = eng.runner.step([b.StepEntry("a", toks, list(range(len(toks))))]).double().cpu()
    assert eng.runner._waits_unchecked == fast
    eng.runner.check_kernels()
    want = torch.as_tensor(plain.forward(*plain.read_model_folder(str(tmp_path)), toks)).double()
    assert ((got - want).norm() / want.norm()) < 2e-6      # sums of up to 384 in 32 bits, two layers


@pytest.mark.parametrize("N,K", [(128, 256), (896, 900), (512, 2048)])
@pytest.mark.parametrize("M", [1, 20, 200])
def test_32_bit_product_of_rows_with_few_numbers(M, N, K):
    """A row of one 1 gives a column of W as it is. Rows of 1, 4 and 16 numbers and full ones: every single result within what a chain of
    as many FMAs is off by at most (half a last place of the sum of magnitudes each; 2 % for the products left out and what follows),
    and the rows' error together no larger than the chain's."""
    o = ops()
    g = torch.Generator().manual_seed(M * 31 + N + K)
    w = (torch.randn(N, K, generator=g) * 0.3).to(DEV)
    out = torch.empty(M, N, device=DEV)
    at = torch.randint(0, K, (M,), generator=g)
    one = torch.zeros(M, K)
    one[torch.arange(M), at] = 1.0
    o.gemm(one.to(DEV), w, out)
    assert torch.equal(out, w[:, at.to(DEV)].T)
    for n in (1, 4, 16, K):
        keep = torch.rand(M, K, generator=g).argsort(dim=1) < n
        x = (torch.randn(M, K, generator=g) * keep).to(DEV)
        o.gemm(x, w, out)
        want, size = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
        assert ((out.double() - want).abs() <= 1.02 * n * 2.0 ** -24 * size).all()
        assert (out.double() - want).norm() <= 1.02 * (fma_chain(x, w).double() - want).norm()
    o.check_status()


def test_32_bit_product_of_tiny_numbers():
    """Operands down to the smallest 32-bit numbers (with large ones on the other side, too) lose no more than in a chain of FMAs, and a
    row's bits are the same beside such rows as without them."""
    o = ops()
    g = torch.Generator().manual_seed(9)
    M, N, K = 40, 256, 512
    x, w = torch.randn(M, K, generator=g).to(DEV), torch.randn(N, K, generator=g).to(DEV)
    before = torch.empty(M, N, device=DEV)
    o.gemm(x, w, before)
    y, v = x.clone(), w.clone()
    scales = {3: 2.0 ** -60, 4: 2.0 ** -112, 5: 2.0 ** -120, 6: 2.0 ** -126, 7: 2.0 ** -140}
    for r, scale in scales.items():
        y[r] *= scale
        v[r] *= scale
    y[8] = 0.0
    y[8, 100] = 2.0 ** -120                            # one number: 2^-120 times a column of W
    y[9] = 0.0
    y[9, 101], y[9, 102] = 2.0 ** -125, 2.0 ** 50      # tiny and huge in one row
    v[10] = 0.0
    v[10, 101] = 2.0 ** 100
    y[11, ::7] = 2.0 ** -130                           # tiny numbers among ordinary ones
    y[12] *= 2.0 ** 45
    out = torch.empty(M, N, device=DEV)
    o.gemm(y, v, out)
    want, chain = y.double() @ v.double().T, fma_chain(y, v)
    # a chain's results are rounded to multiples of 2^-149 where they are that small: what both sides are held to
    size = y.double().abs() @ v.double().abs().T
    for r in [*scales, 8, 9, 11, 12]:
        for c in ([n for n in range(N) if n not in scales], list(scales)):
            err, limit = (out[r, c].double() - want[r, c]).norm(), (chain[r, c].double() - want[r, c]).norm()
            assert err <= 1.02 * limit + 2.0 ** -30 * size[r, c].norm() / K ** 0.5, (r, len(c), err.item(), limit.item())
    assert torch.equal(out[8], chain[8])
    plain_rows = [r for r in range(M) if r not in scales and not 8 <= r <= 12]
    plain_cols = [n for n in range(N) if n not in scales and n != 10]
    assert torch.equal(out[plain_rows][:, plain_cols], before[plain_rows][:, plain_cols])
    alone = torch.empty(1, N, device=DEV)
    for r in (0, 4, 9, 11):
        o.gemm(y[r:r + 1].contiguous(), v, alone)
        assert torch.equal(alone[0], out[r]), r
    o.check_status()


@pytest.mark.parametrize("H,KV,dh,dv,page", [(14, 2, 64, 64, 16), (9, 1, 32, 16, 16), (10, 2, 128, 64, 8), (12, 2, 16, 128, 16), (9, 1, 36, 20, 16), (5, 5, 64, 64, 16)])
@pytest.mark.parametrize("window,extras", [(0, False), (40, True)])
def test_32_bit_attention_with_several_heads_a_warp(H, KV, dh, dv, page, window, extras):
    """Many rows (several heads a warp) against the same rows a few at a time (a warp per head), bit for bit; and against 64 bits."""
    o = ops()
    ctx_lens, q_lens = [211, 1, 64, 300], [211, 1, 33, 170]
    s = paged_setup(ctx_lens, q_lens, KV, dh, page, torch.float32, 3)
    T = s["T"]
    s["kc"] = data(s["kc"].shape, 1)
    vc = data(s["kc"].shape[:3] + (dv,), 2)
    q = data((T, H * dh), 3)
    sinks, gate = (data((H,), 4), data((T, H * dv), 5)) if extras else (None, None)
    cap = 20.0 if extras else 0.0

    def run(t0, t1):
        out = torch.full((t1 - t0, H * dv), float("nan"), device=DEV)
        o.attention_plain(q[t0:t1].contiguous(), s["kc"], vc, s["tok_req"][t0:t1].contiguous(), s["cu_q"] - t0, s["ctx_len"], s["table"], out, H, window,
                          0.3, sinks, None if gate is None else gate[t0:t1], softcap=cap, gate_dim=dv if extras else 0)
        return out
    got = run(0, T)
    few = torch.cat([run(t, min(t + 40, T)) for t in range(0, T, 40)])
    assert T * H >= 2048 > 40 * H and torch.equal(got, few)
    for t in (0, 100, 211, 212, 244, T - 1):
        r, pos = int(s["tok_req_np"][t]), int(s["positions_np"][t])
        j = np.arange(max(0, pos - window + 1) if window else 0, pos + 1)
        pages = torch.from_numpy(s["table_np"][r, j // page]).long().to(DEV)
        k64, v64 = (c[pages, :, torch.from_numpy(j % page).to(DEV)].double() for c in (s["kc"], vc))
        for h in (0, H - 1):
            g = h // (H // KV)
            sc = k64[:, g] @ q[t, h * dh:(h + 1) * dh].double() * 0.3
            if extras:
                sc = torch.cat([cap * torch.tanh(sc / cap), sinks[h:h + 1].double()])
            want = torch.softmax(sc, 0)[:len(j)] @ v64[:, g]
            if extras:
                want = want * torch.sigmoid(gate[t, h * dv:(h + 1) * dv].double())
            close(got[t, h * dv:(h + 1) * dv], want, torch.float32, f"token {t} head {h}")


@pytest.mark.parametrize("K", [4, 16, 20, 36, 64])
@pytest.mark.parametrize("M,N", [(1, 1), (8, 130), (37, 256), (700, 100)])
def test_products_with_a_short_k(M, N, K):
    """Every epilogue, both kinds of W, rows of x in a wider matrix; the same bits for a row alone."""
    o = ops()
    x = data((M, K + 8), 1)[:, :K]
    coef, bias = data((N,), 4).abs() + 0.1, data((N,), 3)
    for wd in (torch.float32, BF):
        w = (data((N, K), 2) * 0.3).to(wd)
        z = x.double() @ w.double().T
        out, one = torch.empty(M, N, device=DEV), torch.empty(1, N, device=DEV)
        o.gemm_plain_decay(x, w, bias, coef, 1, -1.0, out)
        close(out, torch.exp(-coef.double() * torch.nn.functional.softplus(-(z + bias.double()))), torch.float32, "decay")
        o.gemm_plain_decay(x[M // 2:M // 2 + 1], w, bias, coef, 1, -1.0, one)
        assert torch.equal(one[0], out[M // 2])
        o.gemm_plain_decay_exp(x, w, None, out, x_tanh=True)
        close(out, torch.exp(-torch.exp(torch.tanh(x.double()) @ w.double().T)), torch.float32, "decay of exp")
        if wd == BF:
            o.gemm_plain(x, w, out)
            close(out, z, torch.float32, "product")
            o.gemm_plain(x, w, out, bias, o.EPI_BIAS)
            close(out, z + bias.double(), torch.float32, "bias")


@pytest.mark.parametrize("d", [4, 508, 516, 1028, 2052, 4096])
def test_layer_end_chain_of_many_rows(d):
    """More rows than run at once with every operand in registers against the same rows a few at a time, bit for bit."""
    o = ops()
    rows, n = 303, 5
    whole = data((n + 1, rows, d), 61) * 2
    sub, gate, gb = data((rows, d), 62), data((rows, d), 63), data((d,), 64).to(BF)
    pw, pb, tw, tb = ((data((d,), 65 + i) * 0.25 + 1).to(BF) for i in range(4))
    c = data((n,), 70)
    parts = [whole[:, i:i + 100].contiguous() for i in range(0, rows, 100)]
    ys = []
    for i, s in enumerate([whole] + parts):
        r = slice(0, rows) if i == 0 else slice(100 * (i - 1), min(100 * i, rows))
        y = torch.empty(s.shape[1], d, dtype=BF, device=DEV)
        o.norm_chain(s[n - 1], sub[r], gate[r], gb, (pw, pb, 1e-6), streams=s, coeffs=c, n=n, mix_out=s[n], then=(tw, tb, 1e-5), y=y)
        ys.append(y)
    assert torch.equal(whole, torch.cat(parts, dim=1)) and torch.equal(ys[0], torch.cat(ys[1:]))


@pytest.mark.parametrize("dk,dv,rot_half,per", [(8, 8, 4, 1), (64, 128, 32, 2), (64, 64, 16, 1), (128, 64, 64, 3)])
def test_rotation_of_neighbouring_pairs_four_values_at_a_time(dk, dv, rot_half, per):
    """Norms of the q and k rows, neighbours rotated (a part of each head among them), caches written, against 64 bits."""
    o = ops()
    T, KV, page = 9, 2, 16
    H = KV * per
    off_k, off_v = H * dk + 4, (H + KV) * dk + 8
    proj = data((T, off_v + KV * dv + 4), 1) * 2
    qw, kw = data((H * dk,), 2).to(BF), data((KV * dk,), 3)
    pos = torch.tensor([0, 1, 2, 3, 17, 40, 5, 6, 31], dtype=torch.int32, device=DEV)
    req = torch.tensor([0, 0, 0, 0, 0, 0, 1, 1, 1], dtype=torch.int32, device=DEV)
    table = torch.tensor([[3, 0, 5], [1, 4, 2]], dtype=torch.int32, device=DEV)
    inv = torch.from_numpy((1e4 ** (-np.arange(rot_half) / rot_half)).astype(np.float32)).to(DEV)
    q = torch.empty(T, H * dk, device=DEV)
    kc, vc = torch.zeros(6, KV, page, dk, device=DEV), torch.zeros(6, KV, page, dv, device=DEV)
    o.qk_norm_rope_write(proj, off_k, off_v, qw, kw, 1e-6, pos, req, table, inv, rot_half, 1, q, kc, vc, H, KV, dk, dv)
    p64 = proj.double()
    ang = (pos.float()[:, None] * inv).double()[:, None]

    def turned(z, w, heads):
        z = (z / torch.sqrt((z * z).mean(-1, keepdim=True) + 1e-6) * w.double()).view(T, heads, dk)
        a, b = z[..., 0:2 * rot_half:2], z[..., 1:2 * rot_half:2]
        r = torch.stack((a * ang.cos() - b * ang.sin(), b * ang.cos() + a * ang.sin()), -1).flatten(-2)
        return torch.cat([r, z[..., 2 * rot_half:]], -1)
    close(q, turned(p64[:, :H * dk], qw, H).reshape(T, -1), torch.float32, "q")
    pages, rows = table[req.long(), pos.long() // page].long(), pos.long() % page
    close(kc[pages, :, rows], turned(p64[:, off_k:off_k + KV * dk], kw, KV), torch.float32, "k")
    assert torch.equal(vc[pages, :, rows], proj[:, off_v:off_v + KV * dv].view(T, KV, dv))


@pytest.mark.parametrize("unit,dk,C", [(3, 16, 96), (4, 64, 260), (0, 16, 36), (24, 128, 3100)])
def test_short_convolution_of_many_tokens(unit, dk, C):
    """Several tokens a block against a token a block, bit for bit: requests that begin, end and have one token anywhere in a block."""
    o = ops()
    lens = [5, 1, 1, 1, 0, 2, 400, 3, 2, 1, 190, 6]
    T, R = sum(lens), len(lens)
    x, tail = data((T, C + 4), 3), data((R, 3 * C + 4), 5)
    w, bias = data((C, 4), 7), data((C,), 8)
    slots = torch.arange(R, dtype=torch.int32, device=DEV).flip(0).contiguous()
    cu = torch.tensor([0] + lens, device=DEV).cumsum(0).to(torch.int32)
    req = torch.repeat_interleave(torch.arange(R), torch.tensor(lens)).to(torch.int32).to(DEV)
    assert T >= 592
    y = torch.full((T, C), float("nan"), device=DEV)
    o.conv_silu_unit(x, w, tail, slots, req, cu, y, unit, min(unit, 1), dk, 0.25, 1e-6, bias=bias)
    few = torch.full((T, C), float("nan"), device=DEV)
    for r in range(R):                                 # a request by itself
        lo, hi = int(cu[r]), int(cu[r + 1])
        if lo == hi:
            continue
        part = torch.full((hi - lo, C), float("nan"), device=DEV)
        one = torch.tensor([0, hi - lo], dtype=torch.int32, device=DEV)
        o.conv_silu_unit(x[lo:hi], w, tail, slots[r:r + 1].contiguous(), torch.zeros(hi - lo, dtype=torch.int32, device=DEV), one, part, unit,
                         min(unit, 1), dk, 0.25, 1e-6, bias=bias)
        few[lo:hi] = part
    assert torch.equal(y, few)


@pytest.mark.parametrize("H,dv", [(1, 4), (3, 128), (2, 132), (5, 256), (2, 512)])
@pytest.mark.parametrize("gate", [None, "GATE_SILU", "GATE_SIGMOID"])
def test_norm_of_heads_in_groups_of_four(H, dv, gate):
    o = ops()
    T = 7
    x, g, w, wh = data((T, H * dv), 3) * 2, data((T, H * dv + 4), 4), data((dv,), 5).to(BF), data((H * dv,), 6)
    x64 = x.double().view(T, H, dv)
    n64 = x64 / torch.sqrt((x64 * x64).mean(-1, keepdim=True) + 1e-5)
    gv = None if gate is None else g[:, :H * dv]
    f = 1.0 if gate is None else torch.sigmoid(gv.double()) * (gv.double() if gate == "GATE_SILU" else 1.0)
    for dtype in (torch.float32, BF):
        out = torch.empty(T, H * dv, dtype=dtype, device=DEV)
        o.head_norm_gate(x, w, gv, getattr(o, gate or "GATE_SILU"), 1e-5, out, H, dv)
        close(out, (n64 * w.double()).reshape(T, -1) * f, dtype, "shared weight")
        o.head_norm_gate_ext(x, wh, gv, getattr(o, gate or "GATE_SILU"), 1e-5, out, H, dv)
        close(out, n64.reshape(T, -1) * wh.double() * f, dtype, "weight per head")
@pytest.mark.parametrize("M,N,K", [(1, 130, 72), (16, 896, 4864), (17, 2048, 1096), (33, 257, 200), (64, 1024, 136), (9, 19204, 72), (40, 19101, 128)])
def test_few_rows_with_w_streamed_once(M, N, K):
    """Clusters of every size and tiles in rounds (two accumulators taking turns), remainders of rows, columns and k, each epilogue."""
    o = ops()
    x, w, b = (data((M, K), 1) * 0.5).to(BF), (data((N, K), 2) * 0.2).to(BF), data((N,), 3)
    z = x.double() @ w.double().T
    out = torch.empty(M, N, device=DEV)
    o.gemm_tc_few(x, w, out)
    close(out, z, torch.float32, "product")
    o.gemm_tc_few(x, w, out, b, o.EPI_BIAS)
    close(out, z + b.double(), torch.float32, "bias")
    res = data((M, N), 4)
    want = res.double() + z + b.double()
    o.gemm_tc_few(x, w, res, b, o.EPI_RESIDUAL)
    close(res, want, torch.float32, "residual")
    n = N // 2
    act = torch.empty(M, n, dtype=BF, device=DEV)
    o.gemm_tc_few(x, w[:2 * n].contiguous(), act, None, o.EPI_SWIGLU)
    close(act, plain.silu(z[:, :n]) * z[:, n:2 * n], BF, "swiglu")
    o.gemm_tc_few(x, w[:2 * n].contiguous(), act, o.glu_args(o.GLU_CLAMPED, 0.5, DEV), o.EPI_SWIGLU)
    g, u = z[:, :n].clamp(max=0.5), z[:, n:2 * n].clamp(-0.5, 0.5)
    close(act, g * torch.sigmoid(1.702 * g) * (u + 1), BF, "clamped")
    o.check_status()


@pytest.mark.parametrize("kind", ["silu", "gelu", "clamped"])
def test_gated_activation_of_few_rows_is_the_same_in_both_kernels(kind):
    """Sums that are one number of W each (rows of one 1): the two kernels that a gated product of few rows may run on round the same
    activation, bit for bit."""
    o = ops()
    K, N = 256, 4096
    x = torch.zeros(16, K, dtype=BF, device=DEV)
    x[torch.arange(16), torch.arange(16) * 9] = 1.0
    w = (data((2 * N, K), 2) * 8).to(BF)
    act = {"silu": None, "gelu": o.glu_args(o.GLU_GELU_TANH, 0.0, DEV), "clamped": o.glu_args(o.GLU_CLAMPED, 7.0, DEV)}[kind]
    a, b = torch.empty(16, N, dtype=BF, device=DEV), torch.empty(16, N, dtype=BF, device=DEV)
    o.gemm_tc_few(x, w, a, act, o.EPI_SWIGLU)
    o.gemm_skinny(x, w, b, act, o.EPI_SWIGLU)
    o.check_status()
    assert torch.equal(a, b)


def test_few_rows_go_by_the_bytes_of_w():
    """The kernel on either side of its lines (by bytes, and by the share of the device that its blocks fill), and that a product that an RMS norm links to another stays where the norm is."""
    o = ops()
    m = lambda *s: torch.empty(*s, dtype=BF, device=DEV)
    kinds = [(8, 8208, 2048, o.EPI_NONE, "few"), (8, 2560, 2048, o.EPI_BIAS, "skinny"), (16, 2560, 2048, o.EPI_BIAS, "few"), (16, 2048, 2048, o.EPI_RESIDUAL, "skinny"),
             (17, 896, 4864, o.EPI_RESIDUAL, "few"), (64, 896, 4864, o.EPI_RESIDUAL, "splitk"), (64, 3600, 896, o.EPI_NONE, "few"), (64, 1152, 896, o.EPI_BIAS, "skinny"), (64, 11008, 2048, o.EPI_NONE, "tc"),
             (16, 11008, 2048, o.EPI_SWIGLU, "few"), (32, 11008, 2048, o.EPI_SWIGLU, "tc"), (65, 8208, 2048, o.EPI_NONE, "splitk"),
             (8, 1024, 14336, o.EPI_RESIDUAL, "skinny"), (8, 2048, 8192, o.EPI_RESIDUAL, "skinny"), (16, 4608, 1024, o.EPI_RESIDUAL, "skinny"),
             (24, 576, 14336, o.EPI_RESIDUAL, "splitk"), (64, 6144, 14336, o.EPI_RESIDUAL, "splitk"), (64, 8192, 14336, o.EPI_RESIDUAL, "few"),
             (16, 25000, 1024, o.EPI_NONE, "cols"), (16, 18944, 1024, o.EPI_NONE, "few"), (8, 11008, 11008, o.EPI_RESIDUAL, "tc"),
             (24, 11008, 3584, o.EPI_SWIGLU, "tc"), (24, 18944, 3584, o.EPI_SWIGLU, "few"), (32, 3584, 5120, o.EPI_SWIGLU, "tc")]
    for M, N, K, epi, kind in kinds:
        b = torch.empty(N, device=DEV) if epi == o.EPI_BIAS else None
        assert o.gemm_kernel(m(M, K), m(2 * N if epi == o.EPI_SWIGLU else N, K), N, b, epi) == kind, (M, N, K)
    x, w = m(8, 11008), m(2048, 11008)
    assert o.gemm_kernel(x, w, 2048, None, o.EPI_RESIDUAL) == "few" and o.gemm_skinny_links_norm(x, w, 2048, o.EPI_RESIDUAL)


@pytest.mark.parametrize("rule", ["RULE_GLA", "RULE_DELTA", "RULE_BONUS"])
@pytest.mark.parametrize("H,dk,dv", [(1, 16, 36), (2, 32, 132), (1, 64, 128), (1, 48, 20), (2, 128, 68), (1, 256, 32), (1, 512, 24)])
def test_scan_with_four_columns_a_lane(rule, H, dk, dv):
    """Many requests side by side (four columns a lane) against the same taken as few (one column), bit for bit, over the numbers of
    lanes that share a column; columns that end within a block; and against 64 bits."""
    o = ops()
    rule = getattr(o, rule)
    lens = [3, 1, 2, 0, 5, 17] * 100
    T, R = sum(lens), len(lens)
    q, k, v, b = data((T, H * dk), 1) * 0.3, data((T, H * dk), 2) * 0.1, data((T, H * dv), 3), data((T, H), 4)
    a = torch.sigmoid(data((T, H * dk), 5) + 3.0)
    cu = torch.tensor([0] + lens, device=DEV).cumsum(0).to(torch.int32)
    got = []
    for busy in (1, R):
        st, out = data((R, H * dk * dv), 6), torch.full((T, H * dv), float("nan"), device=DEV)
        o.recurrent_scan(rule, q, k, v, a, None if rule == o.RULE_GLA else b, 0.5, st, torch.arange(R, dtype=torch.int32, device=DEV), cu, out,
                         H, H, dk, dv, busy=busy)
        got.append((out, st))
    assert all(torch.equal(x, y) for x, y in zip(*got))
    out, st = got[1]
    first = data((R, H * dk * dv), 6)
    for r in (0, 5, R - 1):
        lo, hi = int(cu[r]), int(cu[r + 1])
        S = first[r].double().view(H, dk, dv)
        w = _scan64(rule, *(x[lo:hi].double().view(hi - lo, H, -1) for x in (q, k, v, a)), b[lo:hi].double(), 0.5, S, H)
        close(out[lo:hi], w.reshape(hi - lo, -1), torch.float32, f"outputs of request {r}")
        close(st[r], S.reshape(-1), torch.float32, f"state of request {r}")


@pytest.mark.parametrize("rule", ["RULE_GLA", "RULE_DELTA", "RULE_BONUS"])
def test_cut_scan_with_scratch_that_is_not_aligned(rule):
    """The parts' states at an address that is no multiple of 16: served by the build that reads them a value at a time, or refused (the
    delta rule, whose folds read transitions in pieces of 16 bytes)."""
    import ctypes
    o = ops()
    rule = getattr(o, rule)
    H, dk, dv, T, parts = 8, 64, 128, 2100, 60
    q, k, v, b = data((T, H * dk), 1) * 0.3, data((T, H * dk), 2) * 0.1, data((T, H * dv), 3), data((T, H), 4)
    a = torch.sigmoid(data((T, H * dk), 5) + 3.0)
    cu, slots = torch.tensor([0, T], dtype=torch.int32, device=DEV), torch.zeros(1, dtype=torch.int32, device=DEV)
    beta = None if rule == o.RULE_GLA else b
    lib = o._lib()
    lib.bl_recurrent_scan_parts_scratch.restype = ctypes.c_longlong
    n = int(lib.bl_recurrent_scan_parts_scratch(rule, 1, 1, parts, H, dk, dv))
    got = []
    for off in (0, 1):
        st, out = data((1, H * dk * dv), 6), torch.full((T, H * dv), float("nan"), device=DEV)
        room = torch.empty(n + 4, device=DEV)[off:]
        call = lambda: o._call(lib.bl_recurrent_scan_parts, rule, o._p(q), H * dk, o._p(k), H * dk, o._p(v), H * dv, o._p(a), H * dk, o._p(beta),
                H if beta is not None else 0, ctypes.c_float(0.5), o._p(st), ctypes.c_longlong(H * dk * dv), o._p(slots), o._p(cu), 1, o._p(out),
                H, H, dk, dv, parts, 1, 1, ctypes.c_void_p(room.data_ptr()), o._stream())
        if off and rule == o.RULE_DELTA:
            with pytest.raises(o.KernelError, match="aligned"):
                call()
            return
        call()
        got.append((out, st))
    for x, y in zip(*got):
        assert ((x - y).norm() / x.norm()) < 1e-5


@pytest.mark.parametrize("H,KV,dh,window", [(14, 2, 64, 0), (4, 4, 64, 100), (16, 2, 128, 0)])
def test_prompts_and_single_tokens_side_by_side(H, KV, dh, window):
    """The two attention launches of a mixed step with the word between them against the same without it, bit for bit, kernel by
    kernel and replayed from a graph in which the queries are written before and the results read behind them, layer after layer."""
    o = ops()
    ctx_lens, q_lens = [700, 90, 3000, 1, 513, 257, 64], [700, 1, 1, 1, 130, 1, 1]
    s = paged_setup(ctx_lens, q_lens, KV, dh, 16, BF, 5)
    s["kc"], s["vc"] = data(s["kc"].shape, 1).to(BF), data(s["vc"].shape, 2).to(BF)
    T = s["T"]
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    tiles = i32([[r, t] for r, n in enumerate(q_lens) if n > 1 for t in range(0, n, 128)])
    singles = i32([r for r, n in enumerate(q_lens) if n == 1])
    src = [data((T, H * dh), 3 + i) for i in range(3)]
    word = torch.zeros(1, dtype=torch.int32, device=DEV)
    splits = o.attention_decode_tma_splits(singles.shape[0], KV, H // KV, dh, 3000)

    def layers(started):
        outs, q = [], torch.empty(T, H * dh, dtype=BF, device=DEV)
        for i in range(6):
            o.cast_rows(src[i % 3], q)
            out = torch.full((T, H * dh), float("nan"), dtype=BF, device=DEV) if i == 0 else torch.empty(T, H * dh, dtype=BF, device=DEV)
            o.attention_prefill_tc(q, s["kc"], s["vc"], s["cu_q"], s["ctx_len"], s["table"], tiles, out, H, window, 0.1, started=started)
            o.attention_decode_tma(q, s["kc"], s["vc"], s["cu_q"], s["ctx_len"], s["table"], singles, splits, out, H, window, 0.1, started=started)
            outs.append(out.float())
        return outs
    want = layers(None)
    assert all(torch.isfinite(w).all() for w in want)
    for _ in range(3):
        assert all(torch.equal(a, b) for a, b in zip(layers(word), want)) and word.item() == 0
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = layers(word)
    for _ in range(5):
        for g in got:
            g.zero_()
        graph.replay()
        assert all(torch.equal(a, b) for a, b in zip(got, want)) and word.item() == 0
    o.check_status()


@pytest.mark.parametrize("K, N", [(256, 192), (200, 72), (8, 8), (1216, 100)])
@pytest.mark.parametrize("T, E, top, spread", [(1, 3, 2, "even"), (50, 4, 2, "even"), (300, 4, 1, "one"), (700, 3, 2, "skewed"), (1030, 16, 2, "even")])
def test_products_of_routed_experts_in_chunks(K, N, T, E, top, spread):
    """`gemm_experts` behind `moe_chunks`, gated and plain, against float64: experts without rows, one expert with all (several chunks),
    shares of every size modulo 16, inner sizes and columns that are not multiples of a tile. A 32-bit sum of K products of bfloat16
    values is off by at most K eps times the sum of their sizes; the gated result is rounded to bfloat16 (2^-8) once more."""
    o = ops()
    g = torch.Generator().manual_seed(T + K)
    if spread == "one":
        ids = torch.full((T, 1), 2, dtype=torch.int32)
    else:
        p = torch.ones(E) if spread == "even" else torch.tensor([0.9, 0.09, 0.01][:E])
        ids = torch.stack([torch.multinomial(p, top, generator=g) for _ in range(T)]).int()
    x = (torch.randn(T, K, generator=g) * 0.5).bfloat16()
    w = (torch.randn(E, 2 * N, K, generator=g) * 0.2).bfloat16()
    pos, row_src, chunks = o.moe_chunks(ids.to(DEV), E)
    assert row_src.numel() == (-(-T * top // 16) + E) * 16
    at = pos.long().cpu()
    assert torch.equal(row_src.cpu()[at], torch.arange(T * top, dtype=torch.int32)) and int((row_src >= 0).sum()) == T * top
    rows = torch.empty((row_src.numel(), K), dtype=BF, device=DEV)
    o.gather_rows(x.to(DEV), row_src, top, rows)
    e, t = ids.flatten().long(), torch.arange(T).repeat_interleave(top)
    full = torch.empty(T * top, 2 * N, dtype=torch.float64)
    size = torch.empty(T * top, 2 * N, dtype=torch.float64)
    for k in range(E):
        mine = e == k
        full[mine] = x[t[mine]].double() @ w[k].double().T
        size[mine] = x[t[mine]].double().abs() @ w[k].double().abs().T
    off = K * 2.0 ** -23 * size
    y = torch.empty((row_src.numel(), 2 * N), dtype=torch.float32, device=DEV)
    o.gemm_experts(rows, w.to(DEV), chunks, y)
    assert ((y[pos.long()].double().cpu() - full).abs() <= off + 1e-30).all()
    act = torch.empty((row_src.numel(), N), dtype=BF, device=DEV)
    o.gemm_experts(rows, w.to(DEV), chunks, act, o.EPI_SWIGLU)
    want = full[:, :N] * torch.sigmoid(full[:, :N]) * full[:, N:]
    slack = 1.1 * off[:, :N] * full[:, N:].abs() + full[:, :N].abs() * off[:, N:] + 1e-5 * want.abs()     # |silu'| <= 1.1; the sigmoid's own error
    assert ((act[pos.long()].double().cpu() - want).abs() <= slack + 2.0 ** -8 * want.abs() + 1e-30).all()
    o.check_status()
