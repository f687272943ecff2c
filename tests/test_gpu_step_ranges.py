"""Kernels of a step at the edges of their ranges: first and last sizes of a tile or a dispatch rule, remainders, odd sizes."""
import math

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from vox_serve_b200 import ops as o

    return o


def _i32(v):
    return torch.tensor(v, dtype=torch.int32, device="cuda")


@pytest.mark.parametrize("new,old,pad", [
    ([1], [0], 0), ([3, 0, 5, 0, 0, 2], [0, 4, 15, 0, 16, 33], 7), ([0, 0, 9], [3, 0, 0], 0), ([1024], [5], 0), ([1025, 1], [0, 0], 3),
    ([1] * 1023 + [0], [7] * 1024, 1), ([2, 1] * 600, [1, 40] * 600, 24),      # request tables on both sides of the one in shared memory
])
def test_plan_rows_prefill(ops, new, old, pad):
    page, chunk, n = 16, 16, len(new)
    kv = [max(a + b, 1) for a, b in zip(new, old)]
    pages = [(x + page - 1) // page for x in kv]
    qo, ip = np.concatenate([[0], np.cumsum(new)]).tolist(), np.concatenate([[0], np.cumsum(pages)]).tolist()
    idx = np.random.RandomState(n).permutation(ip[-1]).tolist()
    T = qo[-1]
    plan = ops.RowPlan(T + pad, "cuda")
    ops.plan_rows(plan, _i32(qo), _i32(ip), _i32(idx), _i32([(x - 1) % page + 1 for x in kv]), n, T + pad, page, chunk)
    req, at = [], []
    for r in range(n):
        req += [r] * new[r]
        at += [kv[r] - new[r] + j for j in range(new[r])]
    assert plan.row_req[:T + pad].tolist() == req + [-1] * pad
    assert plan.row_kvlen[:T + pad].tolist() == [g + 1 for g in at] + [0] * pad
    assert plan.row_page[:T + pad].tolist() == [idx[ip[r] + g // page] for r, g in zip(req, at)] + [-1] * pad
    assert plan.row_slot[:T].tolist() == [g % page for g in at]
    assert plan.row_pagebase[:T].tolist() == [ip[r] for r in req] and plan.row_old[:T].tolist() == [kv[r] - new[r] for r in req]
    chunks = [(g + chunk) // chunk for g in at] + [0] * pad
    assert plan.row_chunk_start[:T + pad + 1].tolist() == [0] + np.cumsum(chunks).tolist()


def _tiled(ops, x):
    """x in the tiled activation layout, written through its index formula"""
    T, K = x.shape
    t = ops.TiledAct(T, K, "cuda")
    n, kb = t.t_tile, (K + 63) // 64
    r, k = torch.arange(T, device="cuda")[:, None], torch.arange(K, device="cuda")[None]
    at = (((r // n) * kb + (k >> 6)) * n + r % n) * 64 + ((((k >> 3) & 7) ^ (r % n & 7)) << 3) + (k & 7)
    t.data[at.reshape(-1)] = x.reshape(-1)
    return t


def _close(got, ref, bound):
    err = ((got.double() - ref).norm() / ref.norm()).item()
    assert err < bound, err


# rows: first one of the kernel for pairs of SMs, its 16-row remainders, one block of the tiled layout and one row more, three
# blocks; weight rows: one tile, an odd number of tiles (the last pair half empty), tile heights with 1, 2 and 4 tiles per CTA;
# k: a remainder of the 64-k blocks, odd numbers of blocks per 128-k stage, more than the ring holds
@pytest.mark.parametrize("T,N,K,tile_rows", [(65, 128, 64, 128), (96, 384, 200, 128), (133, 640, 704, 64), (255, 96, 192, 32),
                                             (256, 480, 320, 96), (257, 1280, 1096, 128), (529, 960, 512, 96), (777, 448, 576, 64)])
def test_wide_projection(ops, T, N, K, tile_rows):
    g = torch.Generator(device="cuda").manual_seed(T)
    x = torch.randn(T, K, generator=g, device="cuda").bfloat16()
    w = (torch.randn(N, K, generator=g, device="cuda") * K ** -0.5).bfloat16()
    b = torch.randn(N, generator=g, device="cuda").bfloat16()
    ref = x.double() @ w.double().T
    pw = ops.pack_weight(w, tile_rows)
    for xin in (x, _tiled(ops, x)):
        for split in (1, min(3, (K + 63) // 64)):
            p = ops.gemm(xin, pw, mode=1, split_k=split, tile_rows=tile_rows, out=torch.full((split, T, N), float("nan"), device="cuda"))
            _close(p.sum(0), ref, 2e-6)                       # 32-bit sums: 2^-24 times the square root of the terms
        y = ops.gemm(xin, pw, mode=0, tile_rows=tile_rows, bias=b, act="relu2", out=torch.full((T, N), float("nan"), device="cuda").bfloat16())
        _close(y, torch.relu(ref + b.double()) ** 2, 2 ** -8)   # one rounding to bf16
    if N % 64 == 0 and (N // 2) % (tile_rows // 2) == 0:
        gate, up = w[:N // 2].contiguous(), w[N // 2:].contiguous()
        gu = ops.pack_weight(ops.interleave_gate_up(gate, up, tile_rows // 2), tile_rows)
        ref = torch.nn.functional.silu(x.double() @ gate.double().T) * (x.double() @ up.double().T)
        xt, yt = _tiled(ops, x), ops.TiledAct(T, N // 2, "cuda")
        _close(ops.gemm(x, gu, mode=2, tile_rows=tile_rows, n_out=N // 2), ref, 4 * 2 ** -8)      # gate, up, silu and product rounded
        _close(ops.gemm(xt, gu, mode=2, tile_rows=tile_rows, n_out=N // 2, out=yt).to_rows(), ref, 4 * 2 ** -8)
    from vox_serve_b200 import _lib

    assert _lib.load().vb_gemm_wide_timeouts() == 0


@pytest.mark.parametrize("kind,scale,slope", [("silu", 1.0, 0), ("silu", 40.0, 0), ("silu", 2.0 ** -120, 0), ("glu", 1.0, 1.702), ("glu", 30.0, 1.702),
                                              ("glu", 2.0 ** -92, 2.0 ** 92), ("glu", 2.0 ** -101, 2.0 ** 103)])
def test_wide_gate_quotients(ops, kind, scale, slope):
    """The gate/up epilogue against the same operations one by one, on two million gates: one value of the quotient that is not
    the division's shows as soon as it lies next to where the output's rounding turns."""
    T, N, K = 1024, 2048, 64
    g = torch.Generator(device="cuda").manual_seed(int(scale * 7) + len(kind))
    x = torch.randn(T, K, generator=g, device="cuda").bfloat16()
    gate, up = ((torch.randn(N, K, generator=g, device="cuda") * K ** -0.5 * s).bfloat16() for s in (scale, 1.0))
    gate[:8] = 0.0
    pw = ops.pack_weight(ops.interleave_gate_up(gate, up, 64), 128)
    gt, ut = (ops.gemm(x, ops.pack_weight(w, 128), mode=1)[0] for w in (gate, up))        # fp32 sums in the same order
    if kind == "silu":
        got = ops.gemm(x, pw, mode=2, tile_rows=128, n_out=N)
        gr = gt.bfloat16().float()
        want = ((gr / (1.0 + torch.exp(-gr))).bfloat16().float() * ut.bfloat16().float()).bfloat16()
    else:
        limit = 7.0
        got = ops.gemm_glu(x, pw, torch.empty(T, N, dtype=torch.bfloat16, device="cuda"), limit, slope)
        gr, ur = gt.clamp(max=limit), ut.clamp(-limit, limit)
        want = ((gr / (1.0 + torch.exp(-slope * gr))) * (ur + 1.0)).bfloat16()
    assert torch.equal(got, want), (got != want).sum().item()


@pytest.mark.parametrize("T", [64, 128])
def test_projections_refuse_alike(ops, T):
    """What the one-SM entries refuse is refused for steps of many rows too: a clamp that is not positive, an activation on a grouped
    gated product."""
    from vox_serve_b200._lib import VoxB200Error

    x = torch.randn(T, 64, device="cuda").bfloat16()
    pw = ops.pack_weight(torch.randn(256, 64, device="cuda").bfloat16(), 64)
    out, grp = torch.empty(T, 128, device="cuda").bfloat16(), _i32([0] * (T // 64))
    for limit in (0.0, -1.0, float("nan")):
        with pytest.raises(VoxB200Error):
            ops.gemm_glu(x, pw, out, limit, 1.0)
        with pytest.raises(VoxB200Error):
            ops.gemm_grouped_glu(x, pw, out, 256, 64, 64, grp, 0, limit, 1.0)
    for tiles in (grp, None):
        with pytest.raises(VoxB200Error):
            ops.gemm_grouped(x, pw, out, 2, 256, 64, 64, tiles, act="gelu")
    ops.gemm_glu(x, pw, out, 7.0, 1.0)
    ops.gemm_grouped(x, pw, out, 2, 256, 64, 64, grp)


@pytest.mark.parametrize("groups,tt,N,K", [(1, 128, 256, 128), (3, 128, 320, 456), (5, 64, 128, 192)])
def test_wide_grouped_projection(ops, groups, tt, N, K):
    g = torch.Generator(device="cuda").manual_seed(groups)
    tiles = groups + 2
    x = torch.randn(tiles * tt, K, generator=g, device="cuda").bfloat16()
    w = (torch.randn(groups, N, K, generator=g, device="cuda") * K ** -0.5).bfloat16()
    pw = ops.pack_weight(w.view(groups * N, K), 64)
    grp = [(7 * i) % groups for i in range(tiles)]
    out = torch.full((tiles * tt, N), float("nan"), device="cuda")
    ops.gemm_grouped(x, pw, out, 1, N, K, tt, _i32(grp), group_bytes=ops.weight_tiles_bytes(N, K, 64))
    ref = torch.cat([x[i * tt:(i + 1) * tt].double() @ w[e].double().T for i, e in enumerate(grp)])
    _close(out, ref, 2e-6)


@pytest.mark.parametrize("T,E,top,shared,N,K,skew", [(1, 4, 1, True, 256, 128, False), (17, 3, 2, False, 320, 200, False), (700, 8, 2, True, 512, 256, False),
                                                     (1001, 8, 2, True, 384, 192, True), (513, 70, 4, False, 128, 64, False), (300, 5, 3, True, 256, 128, True)])
@pytest.mark.parametrize("mode,tile_rows", [(0, 128), (1, 128), (2, 96), (2, 64)])
def test_projection_of_tile_tables(ops, T, E, top, shared, N, K, skew, mode, tile_rows):
    """Every row times its expert's weights, with experts that nobody picked and one that everybody did; the shared expert's rows are the tokens."""
    N = N // (2 * tile_rows) * 2 * tile_rows if mode == 2 else N
    N = max(N, 2 * tile_rows) if mode == 2 else N
    g = torch.Generator(device="cuda").manual_seed(T + E + mode)
    G = E + int(shared)
    w, x = torch.randn(G, N, K, generator=g, device="cuda").bfloat16(), torch.randn(T, K, generator=g, device="cuda").bfloat16()
    pick = torch.argsort(torch.rand(T, E, generator=g, device="cuda"), 1)[:, :top].to(torch.int32)
    if skew:                                   # expert 0 for all, the others from the upper half
        pick = torch.cat((torch.zeros(T, 1, device="cuda", dtype=torch.int32), E // 2 + pick[:, :top - 1] % (E - E // 2)), 1)
    idx = pick.contiguous()
    rows = ((T + 15) // 16 * 16 if shared else 0) + T * top + 16 * E
    token, pair = torch.full((rows,), -7, dtype=torch.int32, device="cuda"), torch.zeros(T * top, dtype=torch.int32, device="cuda")
    tiles = torch.zeros(1 + (T * top + 255) // 256 + (T + 255) // 256 + E + 20, 4, dtype=torch.int32, device="cuda")
    ops.moe_group_tiles(idx, T, E, top, shared, token, pair, tiles, ((N, K), (K, N)))
    xs = ops.moe_gather_rows(x, token, torch.zeros(rows, K, dtype=torch.bfloat16, device="cuda"))
    pack = lambda m: ops.pack_weight(ops.interleave_gate_up(m[:N // 2], m[N // 2:], tile_rows // 2) if mode == 2 else m, tile_rows)          # noqa: E731
    packed = [pack(m.contiguous()) for m in w]
    gb = ops.weight_tiles_bytes(N, K, tile_rows)
    whole = ops.PackedWeight(torch.cat([q.data[:gb] for q in packed]), N, K, tile_rows)
    out = torch.full((rows, N // 2 if mode == 2 else N), -1.0, dtype=torch.float32 if mode == 1 else torch.bfloat16, device="cuda")
    ops.gemm_tiles(xs, whole, out, mode, N, K, tiles, group_bytes=gb)
    tab = tiles.cpu()
    n, covered = int(tab[0, 0]), []
    for e, r0, m, _ in tab[1:1 + n].tolist():
        assert 0 < m <= 256 and r0 % 16 == 0
        covered += [(r, e) for r in range(r0, r0 + m)]
    tok = token.cpu()
    assert len(covered) == len(set(r for r, _ in covered)) == T * top + (T if shared else 0) == int((tok >= 0).sum())
    if shared:
        assert tok[:T].tolist() == list(range(T))
    flat = idx.cpu().view(-1).tolist()
    of = dict(covered)
    for i, r in enumerate(pair.tolist()):
        assert tok[r] == i // top and of[r] == flat[i]
    group = torch.tensor([of.get(r, 0) for r in range(rows)], device="cuda")
    for e in range(G):
        r = ((group == e) & (token >= 0)).nonzero()[:, 0]
        y = xs[r].float() @ w[e].float().T
        if mode == 2:
            a, b = y[:, :N // 2].bfloat16().float(), y[:, N // 2:].bfloat16().float()
            y = (a / (1 + torch.exp(-a))).bfloat16().float() * b
        if r.numel():
            d = (out[r].float() - y).abs()
            assert float(d.max()) <= (1e-5 * K ** 0.5 * 4 if mode == 1 else 2 ** -7 * float(y.abs().max()))          # sums of K in 32 bits; one rounding to bf16 beside ties
    assert ops.check_waits() is None


@pytest.mark.parametrize("lens,old", [([64], [0]), ([65], [2]), ([3, 70, 1, 9], [0, 1, 5, 2]), ([8, 8, 8, 100, 2], [0, 0, 3, 7, 0]), ([200], [0])])
@pytest.mark.parametrize("taps,C,act,residual,shift", [(4, 512, "silu", False, 0), (4, 516, "silu", True, 1), (3, 260, None, True, 0), (2, 4, "silu", False, 0)])
def test_short_convolution_rows(ops, lens, old, taps, C, act, residual, shift):
    """Groups of rows inside a request, across its edges, past the end; taps on and off 16-byte boundaries; activations whose quotients leave the short way."""
    g = torch.Generator(device="cuda").manual_seed(sum(lens) + taps)
    rnd = lambda *n: torch.randn(*n, generator=g, device="cuda")          # noqa: E731
    T, B, K = sum(lens), len(lens), taps - 1
    x, w, b, ib = rnd(T, C), rnd(C * taps + shift)[shift:].view(C, taps), rnd(C), rnd(C)
    x[T // 2, :4] = torch.tensor([300.0, -300.0, 1e30, -1e-30], device="cuda")
    state = rnd(B, K, C)
    was, qo = state.clone(), [0]
    for n in lens:
        qo.append(qo[-1] + n)
    req = [i for i, n in enumerate(lens) for _ in range(n)]
    pos = [o + r for n, o in zip(lens, old) for r in range(n)]
    out = torch.empty(T, C, device="cuda")
    ops.short_conv(x, w, b, state, _i32(qo), _i32(req), _i32(pos), _i32(list(range(B))), B, out_f32=out, act=act, residual=residual, in_bias=ib)
    u = x.double() + ib.double()
    for i, n in enumerate(lens):
        at = slice(qo[i], qo[i + 1])
        front = was[i].double().clone()
        front[:max(0, K - old[i])] = 0                      # positions before the first
        full = torch.cat((front, u[at]))
        y = sum(full[j:j + n] * w[:, j].double() for j in range(taps)) + b.double()
        size = sum(full[j:j + n].abs() * w[:, j].double().abs() for j in range(taps)) + b.double().abs()
        # the sum to 2^-22 of its terms; the activation's slope is below 1.1, its exponential and quotient good to a few units
        want, slack = (y * torch.sigmoid(y), 1.1) if act else (y, 1.0)
        if residual:
            want, size = want + u[at], size + u[at].abs()
        assert bool(((out[at].double() - want).abs() <= slack * 1e-6 * size + 1e-37).all())
        assert torch.equal(state[i], torch.cat((front, u[at]))[-K:].float() if n >= K else torch.cat((front.float(), (x + ib)[at]))[-K:])


@pytest.mark.parametrize("taps,act,shift", [(4, "silu", 0), (4, "silu", 1), (3, None, 0), (2, "silu", 0)])
def test_short_convolution_rows_by_twos_and_fours(ops, taps, act, shift):
    """A thread takes two rows or four by the size of the launch: the same bits for a quarter of the channels alone, with requests that begin anywhere in a group."""
    g = torch.Generator(device="cuda").manual_seed(taps)
    lens, old, C = [3, 70, 1, 9, 2, 5, 611], [0, 1, 5, 2, 0, 0, 7], 2048
    T, B = sum(lens), len(lens)
    x, w, bias, state = (torch.randn(*n, generator=g, device="cuda") for n in ((T, C), (C * taps + 1,), (C,), (B, taps - 1, C)))
    w = w[shift:shift + C * taps].view(C, taps)          # (shifted: taps off the 16-byte boundaries)
    plan = (_i32([sum(lens[:i]) for i in range(B + 1)]), _i32([i for i, n in enumerate(lens) for _ in range(n)]),
            _i32([o + k for o, n in zip(old, lens) for k in range(n)]), _i32(list(range(B))), B)

    def run(c):
        st, out, f32 = state[:, :, :c].clone(memory_format=torch.contiguous_format), torch.zeros(T, c, device="cuda", dtype=torch.bfloat16), torch.zeros(T, c, device="cuda")
        ops.short_conv(x[:, :c].contiguous(), w[:c], bias[:c].contiguous(), st, *plan, out=out, out_f32=f32, act=act, residual=True)
        return st, out, f32

    for a, b in zip(run(C), run(C // 4)):
        assert torch.equal(a[..., :C // 4], b)


# channels-last vocoder convolutions: one row and several batch entries in a box, box sizes around 128 rows, a range inside the
# sequence, column tiles with a remainder, dilated taps reaching in front of the start; every epilogue and activation
@pytest.mark.parametrize("B,T,C,N,ksize,dil,lo,hi,epi,act", [
    (1, 1, 32, 32, 1, 1, 0, 1, "plain", None), (7, 16, 64, 96, 1, 1, 0, 16, "resid", "snake"), (2, 128, 32, 128, 3, 1, 0, 128, "plain", "elu"),
    (3, 129, 96, 160, 1, 1, 5, 129, "noise", None), (1, 300, 64, 64, 7, 9, 130, 299, "scale_resid", "gelu"), (40, 3, 128, 512, 2, 1, 0, 3, "resid", None)])
def test_channels_last_conv(B, T, C, N, ksize, dil, lo, hi, epi, act):
    from vox_serve_b200 import _lib
    from vox_serve_b200.tokenizer import _cl

    g = torch.Generator(device="cuda").manual_seed(T + N)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")                 # noqa: E731
    x, w, b, r = rnd(B, T, C), rnd(N, C, ksize) * (C * ksize) ** -0.5, rnd(N), rnd(B, T, N)
    sc, nz, al = rnd(N), rnd(B, T), torch.rand(N, generator=g, device="cuda") + 0.5
    wrap = lambda t: _cl.Act(t.reshape(-1).clone(), B, T, t.shape[-1])           # noqa: E731
    kw = dict(ksize=ksize, dil=dil, epi=epi, resid=None if epi == "plain" else wrap(r), scale=sc, noise=nz, act=act,
              alpha=torch.cat((al, 1 / (al + 1e-9))), lo=lo, hi=hi)
    v = torch.nn.functional.conv1d(torch.nn.functional.pad(x.double().transpose(1, 2), ((ksize - 1) * dil, 0)), w.double(), b.double(),
                                   dilation=dil).transpose(1, 2)
    v = {"plain": v, "resid": r + v, "scale_resid": r + sc * v, "noise": r + nz[..., None] * v}[epi].double()
    z = {None: v, "snake": v + torch.sin(al * v) ** 2 / (al.double() + 1e-9), "elu": torch.nn.functional.elu(v),
         "gelu": torch.nn.functional.gelu(v)}[act]
    _close(_cl.conv(wrap(x), _cl.pack_conv(w.reshape(N, -1), C, ksize), N, b, **kw).tensor()[:, lo:hi], z[:, lo:hi], 5e-6)
    plain, both = _cl.conv(wrap(x), _cl.pack_conv(w.reshape(N, -1), C, ksize), N, b, both=True, **kw)
    _close(plain.tensor()[:, lo:hi], v[:, lo:hi], 5e-6)                          # 32-bit sums of products exact to 2^-22
    _close(both.tensor()[:, lo:hi], z[:, lo:hi], 5e-6)
    assert _lib.load().vb_cl_timeouts() == 0


@pytest.mark.parametrize("B,T,C,N,ksize", [(1, 128, 1024, 128, 7), (3, 40, 256, 32, 3), (160, 128, 64, 64, 3)])
def test_channels_last_conv_reuses_stages(B, T, C, N, ksize):
    """A stage's tensor-memory columns are written again while products of earlier k-blocks may still be running: many turns of the
    ring (long k, and several units per CTA), every run equal to the first bit for bit and to 64 bits."""
    from vox_serve_b200.tokenizer import _cl

    g = torch.Generator(device="cuda").manual_seed(C)
    x, w = torch.randn(B, T, C, generator=g, device="cuda"), torch.randn(N, C, ksize, generator=g, device="cuda") * (C * ksize) ** -0.5
    xa, wp = _cl.Act(x.reshape(-1), B, T, C), _cl.pack_conv(w.reshape(N, -1), C, ksize)
    y = _cl.conv(xa, wp, N, ksize=ksize).tensor()
    ref = torch.nn.functional.conv1d(torch.nn.functional.pad(x.double().transpose(1, 2), (ksize - 1, 0)), w.double()).transpose(1, 2)
    _close(y, ref, 3 * C * ksize / 8 * 2 ** -24)      # each of the 3 K / 8 accumulations cuts off up to 2^-23, half of it on average
    for _ in range(20):
        assert torch.equal(_cl.conv(xa, wp, N, ksize=ksize).tensor(), y)


# tiles of 128 channels and a last one of 32 or 64, three and more units a CTA, so that a CTA goes from one width to the other; without boxes
# (parts, 288) and with them
@pytest.mark.parametrize("T,C,N,ksize", [(32768, 256, 288, 3), (32768, 512, 320, 1), (20000, 512, 544, 1), (9001, 256, 320, 3)])
@pytest.mark.parametrize("parts", [False, True])
def test_channels_last_conv_of_two_tile_widths(T, C, N, ksize, parts):
    from vox_serve_b200 import _lib
    from vox_serve_b200.tokenizer import _cl

    g = torch.Generator(device="cuda").manual_seed(N)
    x, w = torch.randn(1, T, C, generator=g, device="cuda"), torch.randn(N, C, ksize, generator=g, device="cuda") * (C * ksize) ** -0.5
    act = _cl.Act(x.reshape(-1).clone(), 1, T, C)
    if parts:
        act = _cl.conv(act, _cl.pack(torch.eye(C, device="cuda")), C, out="parts")
    ref = torch.nn.functional.conv1d(torch.nn.functional.pad(x.double().transpose(1, 2), (ksize - 1, 0)), w.double()).transpose(1, 2)
    y, z = _cl.conv(act, _cl.pack_conv(w.reshape(N, -1), C, ksize), N, ksize=ksize, act="elu", both=True, out="parts")
    single = _cl.conv(act, _cl.pack_conv(w.reshape(N, -1), C, ksize), N, ksize=ksize).tensor()
    back = _cl.conv(z, _cl.pack(torch.eye(N, device="cuda")), N).tensor()
    err = lambda got, want: (((got.double() - want).norm(dim=2) / want.norm(dim=2)).max()).item()      # noqa: E731  (of the worst position)
    assert err(y.tensor(), ref) < 1e-5 and err(single, ref) < 1e-5 and err(back, torch.nn.functional.elu(ref)) < 1e-5
    assert _lib.load().vb_cl_timeouts() == 0


# activations kept as parts: several entries and their halos in a tile, runs with a remainder, taps further apart than a tile's halo holds, K
# divided over a cluster, boxes of results and none, two results; values of ordinary size, larger than fp16 and all below its normal range
@pytest.mark.parametrize("B,T,C,N,ksize,dil,lo,hi,epi,act,both,size", [
    (1, 1, 32, 32, 1, 1, 0, 1, "plain", None, False, 1.0), (7, 16, 64, 96, 3, 1, 0, 16, "resid", "snake", False, 1.0), (2, 128, 32, 128, 3, 1, 0, 128, "plain", "elu", True, 1.0),
    (3, 129, 96, 160, 2, 1, 5, 129, "noise", None, False, 1.0), (1, 300, 64, 64, 7, 9, 130, 299, "scale_resid", "gelu", False, 1.0),
    (40, 3, 128, 512, 2, 1, 0, 3, "resid", None, True, 1.0), (1, 40, 64, 32, 5, 30, 0, 40, "plain", None, False, 1.0), (1, 17, 1024, 256, 2, 1, 0, 17, "plain", "elu", True, 1.0),
    (3, 700, 64, 128, 1, 1, 0, 700, "resid", "elu", False, 1.0), (2, 900, 128, 256, 2, 1, 3, 899, "plain", "elu", True, 1.0), (2, 50, 64, 64, 3, 1, 0, 50, "resid", "elu", True, 3e5),
    (2, 50, 64, 64, 3, 1, 0, 50, "plain", None, False, 1e-6)])
def test_channels_last_parts(B, T, C, N, ksize, dil, lo, hi, epi, act, both, size):
    from vox_serve_b200 import _lib
    from vox_serve_b200.tokenizer import _cl

    g = torch.Generator(device="cuda").manual_seed(T + N)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")                 # noqa: E731
    x, w, b, r = rnd(B, T, C) * size, rnd(N, C, ksize) * (C * ksize) ** -0.5, rnd(N) * size, rnd(B, T, N) * size
    sc, nz, al = rnd(N), rnd(B, T), torch.rand(N, generator=g, device="cuda") + 0.5
    wrap = lambda t: _cl.Act(t.reshape(-1).clone(), B, T, t.shape[-1])           # noqa: E731
    eye = _cl.pack(torch.eye(C, device="cuda"))
    xp = _cl.conv(wrap(x), eye, C, out="parts")                                  # the values, to the 2^-22 that parts hold
    kw = dict(ksize=ksize, dil=dil, epi=epi, resid=None if epi == "plain" else wrap(r), scale=sc, noise=nz, act=act,
              alpha=torch.cat((al, 1 / (al + 1e-9))), lo=lo, hi=hi)
    v = torch.nn.functional.conv1d(torch.nn.functional.pad(x.double().transpose(1, 2), ((ksize - 1) * dil, 0)), w.double(), b.double(),
                                   dilation=dil).transpose(1, 2)
    v = {"plain": v, "resid": r + v, "scale_resid": r + sc * v, "noise": r + nz[..., None] * v}[epi].double()
    z = {None: v, "snake": v + torch.sin(al * v) ** 2 / (al.double() + 1e-9), "elu": torch.nn.functional.elu(v),
         "gelu": torch.nn.functional.gelu(v)}[act]
    wp = _cl.pack_conv(w.reshape(N, -1), C, ksize)
    _close(_cl.conv(xp, wp, N, b, **kw).tensor()[:, lo:hi], z[:, lo:hi], 5e-6)
    out = _cl.conv(xp, wp, N, b, both=both, out="parts", **kw)                   # what the next convolution reads, through an identity
    plain, out = out if both else (None, out)
    if both:
        _close(plain.tensor()[:, lo:hi], v[:, lo:hi], 5e-6)
    back = _cl.conv(out, _cl.pack(torch.eye(N, device="cuda")), N, lo=lo, hi=hi)
    _close(back.tensor()[:, lo:hi], z[:, lo:hi], 5e-6)
    assert _lib.load().vb_cl_timeouts() == 0


@pytest.mark.parametrize("code", [0x7fffffff, 0x7f800000, 0x7f7fffff])
@pytest.mark.parametrize("C,ksize", [(64, 3), (64, 1)])
def test_channels_last_parts_special_values(code, C, ksize):
    """What parts cannot hold is kept as it is, and reaches the positions and channels that it reaches in fp32, no others."""
    from vox_serve_b200.tokenizer import _cl

    B, T, N = 2, 300, 96
    g = torch.Generator(device="cuda").manual_seed(T)
    x, w = torch.randn(B, T, C, generator=g, device="cuda"), torch.randn(N, C, ksize, generator=g, device="cuda") * 2.0 ** -10
    zero = _cl.Act(torch.zeros(B * T * C, device="cuda"), B, T, C)
    x[1, 133, 37] = _bits(code)
    xp = _cl.conv(zero, _cl.pack(torch.eye(C, device="cuda")), C, epi="resid", resid=_cl.Act(x.reshape(-1).clone(), B, T, C), out="parts")
    y = _cl.conv(xp, _cl.pack_conv(w.reshape(N, -1), C, ksize), N, ksize=ksize).tensor()
    bad = torch.zeros(B, T, N, dtype=torch.bool, device="cuda")
    bad[1, 133:133 + ksize] = True
    if code == 0x7f7fffff:
        ref = torch.nn.functional.conv1d(torch.nn.functional.pad(x.double().transpose(1, 2), (ksize - 1, 0)), w.double()).transpose(1, 2)
        assert torch.isfinite(y).all()
        _close(y[bad], ref[bad], 5e-6)
        _close(y[~bad], ref[~bad], 5e-6)
    else:
        assert torch.equal(~torch.isfinite(y), bad)

def _kept_as_parts(x):
    """x [B, T, C] as parts, exactly where they can hold it: written by the epilogue from a residual"""
    from vox_serve_b200.tokenizer import _cl

    B, T, C = x.shape
    zero = _cl.Act(torch.zeros(B * T * C, device="cuda"), B, T, C)
    return _cl.conv(zero, _cl.pack(torch.eye(C, device="cuda")), C, epi="resid", resid=_cl.Act(x.reshape(-1).clone(), B, T, C), out="parts")


@pytest.mark.parametrize("size", [1.0, 1e-3, 1e-4, 3e-5, 1e-5, 7e-6, 1e-8])
def test_channels_last_parts_hold_22_bits(size):
    """What the next convolution reads of a row is as close to it at every magnitude, beside rows of order one: the second rounding to 11
    bits leaves 4.4e-8 (as two tf32 terms do), the sum of both parts an fp32 rounding."""
    from vox_serve_b200.tokenizer import _cl

    T, C = 512, 64
    x = torch.randn(1, T, C, generator=torch.Generator("cuda").manual_seed(7), device="cuda")
    x[:, ::2] *= size
    y = _cl.conv(_kept_as_parts(x), _cl.pack(torch.eye(C, device="cuda")), C).tensor()
    _close(y[:, ::2], x[:, ::2].double(), 5.5e-8)


# several entries in a tile, flattened rows, a tile of one entry, K divided over a cluster, taps that have stages of their own
_MIXED = [(5, 16, 64, 96, 3, 1), (5, 40, 64, 64, 1, 1), (2, 700, 32, 32, 3, 1), (5, 17, 1024, 256, 2, 1), (3, 130, 128, 64, 5, 30), (1, 500, 64, 128, 1, 1)]


@pytest.mark.parametrize("B,T,C,N,ksize,dil", _MIXED)
@pytest.mark.parametrize("parts", [False, True])
def test_channels_last_conv_of_quiet_passages(B, T, C, N, ksize, dil, parts):
    """Passages of very different magnitude in one tile: each result is as exact as its own inputs let it be."""
    from vox_serve_b200.tokenizer import _cl

    g = torch.Generator(device="cuda").manual_seed(T + N)
    x, w = torch.randn(B, T, C, generator=g, device="cuda"), torch.randn(N, C, ksize, generator=g, device="cuda") * (C * ksize) ** -0.5
    levels = torch.tensor([1.0, 1e-9, 1e-4, 3e4, 1e-7, 1e-5, 0.0], device="cuda")
    run = torch.arange(B * T, device="cuda").view(B, T) // (13 if T < 100 else 61)           # passages that end anywhere in a chunk of rows
    level = run % len(levels)
    x = x * levels[level][..., None]
    act = _kept_as_parts(x) if parts else _cl.Act(x.reshape(-1).clone(), B, T, C)
    y = _cl.conv(act, _cl.pack_conv(w.reshape(N, -1), C, ksize), N, ksize=ksize, dil=dil).tensor().double()
    back = (ksize - 1) * dil
    ref = torch.nn.functional.conv1d(torch.nn.functional.pad(x.double().transpose(1, 2), (back, 0)), w.double(), dilation=dil).transpose(1, 2)
    whole = torch.ones(B, T, dtype=torch.bool, device="cuda")                    # the results of one passage alone
    for s in range(dil, back + 1, dil):
        whole[:, s:] &= run[:, s:] == run[:, :T - s]
    for k, m in enumerate(levels.tolist()):
        sel = whole & (level == k)
        if m == 0.0:
            assert not y[sel].any()
        elif sel.any():
            _close(y[sel], ref[sel], 5e-6)


@pytest.mark.parametrize("B,T,C,N,ksize,dil", [m for m in _MIXED if m[0] == 5] + [(5, 300, 32, 32, 3, 1), (2000, 5, 64, 96, 3, 1)])
@pytest.mark.parametrize("parts", [False, True])
def test_channels_last_conv_alone_and_in_a_batch(B, T, C, N, ksize, dil, parts):
    """An entry's results are the same bits whatever lies beside it: ordinary, quiet, large and silent entries, one that is not a number;
    as floats and as what the next convolution reads."""
    from vox_serve_b200.tokenizer import _cl

    g = torch.Generator(device="cuda").manual_seed(T + C)
    x, w = torch.randn(B, T, C, generator=g, device="cuda"), torch.randn(N, C, ksize, generator=g, device="cuda") * (C * ksize) ** -0.5
    b = torch.randn(N, generator=g, device="cuda") * 1e-3
    x[1::5] *= 1e-9
    x[2::5, T // 2, 5] = math.nan
    x[3::5, T // 3:] *= 3e3
    x[4::5, T // 4:] = 0.0
    wp = _cl.pack_conv(w.reshape(N, -1), C, ksize)

    def run(v):
        """bits of every entry: [plain, activated], [parts, their codes]"""
        n, res = v.shape[0], []
        act = _kept_as_parts(v) if parts else _cl.Act(v.reshape(-1).clone(), n, T, C)
        for out in ("f32", "parts"):
            y, z = _cl.conv(act, wp, N, b, ksize=ksize, dil=dil, act="elu", both=True, out=out)
            res.append([t.buf[:n * T * N].view(torch.int32).view(n, -1) for t in (y, z)])
            if out == "parts":
                res.append([z.buf[n * T * N:].view(torch.uint8)[:n * T * N // 32].view(n, -1)])
        return [torch.cat([t[i].reshape(-1).int() for r in res for t in r]) for i in range(n)]

    together = run(x)
    for i in [*range(5), *range(B - 5, B)]:
        assert torch.equal(together[i], run(x[i:i + 1])[0]), i


def _activated(values, act, alpha=None):
    """The epilogue's activation of given fp32 values: a convolution of zeros with the values as its residual"""
    from vox_serve_b200.tokenizer import _cl

    n = values.numel() // 32
    zero = _cl.Act(torch.zeros(n * 32, device="cuda"), 1, n, 32)
    w = _cl.pack(torch.zeros(32, 32, device="cuda"))
    return _cl.conv(zero, w, 32, epi="resid", resid=_cl.Act(values, 1, n, 32), act=act, alpha=alpha).tensor().reshape(-1).double()


def test_vocoder_activations_over_their_range():
    """The polynomials against 64 bits: ELU down to where it is -1, the squared sine to the end of its reduction and past it."""
    g = torch.Generator(device="cuda").manual_seed(1)
    u = torch.rand(1 << 20, generator=g, device="cuda")
    neg = torch.cat((-90 * u, -2.0 ** (-140 * u), torch.tensor([0.0, -0.0, -80.0, -1e4, 1.5, 3e38] + [0.0] * 26, device="cuda")))
    v = neg.double()
    want = torch.where(v > 0, v, torch.expm1(v))
    got = _activated(neg, "elu")
    assert ((got - want).abs() <= 1e-7 * want.abs() + 2.0 ** -149).all()
    # value + scale sin^2: the scale brings the square to the top of the sum.  Three roundings of a remainder of up to pi / 2
    scale = 2.0 ** 24
    table = torch.cat((torch.ones(32, device="cuda"), torch.full((32,), scale, device="cuda")))
    for top, bound in ((4.0, 5e-7), (65536.0, 5e-7), (1e6, 5e-7)):
        x = (2 * u - 1) * top
        got = (_activated(x, "snake", table) - x.double()) / scale
        assert ((got - torch.sin(x.double()) ** 2).abs() <= bound + x.double().abs() * 2.0 ** -24 / scale).all(), top
    x = 2.0 ** (-20 * u)                                  # small arguments keep their relative accuracy
    got = (_activated(x, "snake", table) - x.double()) / scale
    assert ((got - torch.sin(x.double()) ** 2).abs() <= 5e-7 * torch.sin(x.double()) ** 2 + x.double() * 2.0 ** -23 / scale).all()


@pytest.mark.parametrize("entries,rows,N,far", [(3, 40, 32, (1 << 30) + 64), (1, (1 << 20) + 300, 1024, 0), (2, 150, 64, (1 << 30) - 64)])
def test_channels_last_conv_past_32_bit_offsets(entries, rows, N, far):
    """Batch entries 2^30 floats apart and results of more than 2^30 floats run in several launches."""
    from vox_serve_b200.tokenizer import _cl

    C, B, T = 32, entries, rows
    g = torch.Generator(device="cuda").manual_seed(N)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")                 # noqa: E731
    x, w, b = rnd(B, T, C), rnd(N, C) * C ** -0.5, rnd(N)
    r, nz = (rnd(B, T, N), rnd(B, T)) if far else (None, None)
    y = torch.empty((B - 1) * far + T * N, device="cuda")
    from vox_serve_b200 import ops
    from vox_serve_b200._lib import call

    call("vb_cl_conv", y.data_ptr(), None, x.data_ptr(), T * C, T, _cl.pack(w).data_ptr(), b.data_ptr(), None if r is None else r.data_ptr(), T * N, None,
         None if nz is None else nz.data_ptr(), T, None, 3 if far else 0, 0, B, C, N, N, 1, 1, 0, T, far if far else T * N, ops._stream())
    for i in range(B):
        got = y[i * far:i * far + T * N].view(T, N)
        for c in (slice(0, 200), slice(T - 400 if T > 400 else 0, T)):
            ref = x[i, c].double() @ w.double().T + b.double()
            _close(got[c], ref if r is None else r[i, c] + nz[i, c, None] * ref, 5e-6)


def _bits(*codes):
    return torch.tensor([c - (1 << 32) if c >> 31 else c for c in codes], dtype=torch.int32, device="cuda").view(torch.float32)


# NaN as arithmetic writes it, quiet, negative, with a payload in the bits that tf32 drops; both infinities; the largest finite values
@pytest.mark.parametrize("code,finite", [(0x7fffffff, False), (0x7fc00000, False), (0xffffffff, False), (0x7f800001, False), (0xff801000, False),
                                         (0x7f800000, False), (0xff800000, False), (0x7f7fffff, True), (0xff7ff000, True), (0x7f7fefff, True)])
@pytest.mark.parametrize("where", ["x", "w"])
def test_channels_last_conv_special_values(code, finite, where):
    from vox_serve_b200.tokenizer import _cl

    B, T, C, N, ks = 2, 70, 64, 96, 3
    g = torch.Generator(device="cuda").manual_seed(T)
    x, w = torch.randn(B, T, C, generator=g, device="cuda"), torch.randn(N, C, ks, generator=g, device="cuda") * 2.0 ** -10
    if where == "x":
        x[1, 33, 37] = _bits(code)
        bad = torch.zeros(B, T, N, dtype=torch.bool, device="cuda")
        bad[1, 33:33 + ks] = True
    else:
        x *= 2.0 ** -10
        w[50, 21, 1] = _bits(code)
        bad = torch.zeros(B, T, N, dtype=torch.bool, device="cuda")
        bad[:, :, 50] = True                             # (the first position too: its tap reads the zero in front)
    y = _cl.conv(_cl.Act(x.reshape(-1).clone(), B, T, C), _cl.pack_conv(w.reshape(N, -1), C, ks), N, ksize=ks).tensor()
    if not finite:
        assert torch.equal(~torch.isfinite(y), bad)
        if code & 0x7fffffff != 0x7f800000:
            assert torch.isnan(y[bad]).all()
    else:
        ref = torch.nn.functional.conv1d(torch.nn.functional.pad(x.double().transpose(1, 2), (ks - 1, 0)), w.double()).transpose(1, 2)
        assert torch.isfinite(y).all()
        _close(y[bad], ref[bad], 5e-6)
        _close(y[~bad], ref[~bad], 5e-6)


def test_vocoders_keep_nan(monkeypatch):
    """What is not a number comes out as such, at the positions of the decoders on CUDA cores."""
    from vox_serve_b200.tokenizer.mimi import MimiConfig, MimiDecoder, synthetic_state_dict
    from vox_serve_b200.tokenizer.snac import SNAC

    nan = _bits(0x7fffffff)[0]
    out = []
    for plain in ("0", "1"):
        monkeypatch.setenv("VB_SNAC_FP32", plain)
        m = SNAC(device="cuda")
        sd = m.synthetic_state_dict(3)
        m.load_state_dict(sd)
        assert m.channels_last == (plain == "0")
        m.w["codebooks"][1, 7] = nan
        codes = [torch.zeros(1, n, dtype=torch.int64, device="cuda") for n in (16, 32, 64)]
        codes[1][0, 12] = 7
        noises = [torch.zeros(*s, device="cuda") for s in m.noise_shapes(1, 64)]
        out.append(torch.isnan(m.decode(codes, noises=noises)))
    assert out[0].any() and not out[0].all() and torch.equal(out[0], out[1])

    cfg = MimiConfig(num_layers=2)
    sd = synthetic_state_dict(cfg, 4)
    codes = torch.zeros(2, cfg.n_q, 8, dtype=torch.int64, device="cuda")
    codes[1, 3, 5] = 9
    out = []
    for plain in ("0", "1"):
        monkeypatch.setenv("VB_CODEC_FP32", plain)
        m = MimiDecoder(mimi_config=cfg, state_dict=sd)
        assert m.channels_last == (plain == "0")
        m.w["codebooks"][3, 9] = nan
        out.append(torch.isnan(m.decode(codes)))
    assert not out[0][0].any() and out[0][1].any() and not out[0][1].all() and torch.equal(out[0], out[1])


@pytest.mark.parametrize("B,T,C,cout,s,pad", [(1, 1, 32, 32, 2, 1), (5, 17, 64, 64, 8, 4), (2, 130, 128, 32, 5, 0), (1, 200, 64, 96, 3, 2)])
def test_channels_last_transposed_conv(B, T, C, cout, s, pad):
    from vox_serve_b200.tokenizer import _cl

    g = torch.Generator(device="cuda").manual_seed(T)
    x, w = torch.randn(B, T, C, generator=g, device="cuda"), torch.randn(C, cout, 2 * s, generator=g, device="cuda") * (2 * C) ** -0.5
    b = torch.randn(cout, generator=g, device="cuda")
    wp = w.view(C, cout, 2, s).permute(3, 1, 2, 0).reshape(s, cout, 2 * C)
    y = _cl.conv_transposed(_cl.Act(x.reshape(-1).clone(), B, T, C), _cl.pack_convtr(wp), cout, s, b, pad)
    ref = torch.nn.functional.conv_transpose1d(x.double().transpose(1, 2), w.double(), b.double(), stride=s)[..., pad:pad + T * s]
    _close(y.tensor(), ref.transpose(1, 2), 5e-6)


@pytest.mark.parametrize("B,T,C,dil,lo,hi,big", [(1, 1, 64, 1, 0, 1, 1.0), (3, 65, 128, 3, 0, 65, 1.0), (2, 200, 64, 9, 7, 199, 1.0), (1, 70, 64, 1, 0, 70, 3e5)])
def test_channels_last_depthwise_and_last(B, T, C, dil, lo, hi, big):
    """``big``: arguments of the sine past the range of its reduction (they take the library's)."""
    from vox_serve_b200.tokenizer import _cl

    g = torch.Generator(device="cuda").manual_seed(T)
    x, w = torch.randn(B, T, C, generator=g, device="cuda") * big, torch.randn(C, 7, generator=g, device="cuda")
    b, a1, a2 = (torch.rand(C, generator=g, device="cuda") + 0.5 for _ in range(3))
    table = lambda a: torch.cat((a, 1 / (a + 1e-9)))                             # noqa: E731

    def snake(v, a):                       # (the sine of the 32-bit product: at large arguments its rounding is the result)
        y = (v.float() * a[:, None]).double()
        return v.double() + torch.sin(y) ** 2 / (a.double()[:, None] + 1e-9)

    xs = _cl.Act(x.reshape(-1).clone(), B, T, C)
    y = _cl.depthwise7(xs, w.t().contiguous(), b, table(a1), table(a2) if big == 1.0 else None, dil, lo, hi).tensor()
    v = torch.nn.functional.conv1d(snake(x.transpose(1, 2), a1), w.double()[:, None], b.double(), dilation=dil, padding=3 * dil, groups=C)
    v = snake(v.float(), a2) if big == 1.0 else v
    _close(y[:, lo:hi], v.transpose(1, 2)[:, lo:hi], 5e-6)
    last = _cl.last_conv(xs, w, b[:1], 7, 3, lo, hi, tanh=False)
    ref = torch.nn.functional.conv1d(x.double().transpose(1, 2), w.double()[None], b[:1].double(), padding=3)[..., lo:hi]
    _close(last, ref, 5e-6)


@pytest.mark.parametrize("C,rows,dil", [(64, 1, 1), (512, 15, 9), (512, 17, 1), (256, 33, 3), (256, 97, 64), (320, 129, 9)])
@pytest.mark.parametrize("parts", [False, True])
def test_channels_last_depthwise_tiles(C, rows, dil, parts):
    """A row's result does not depend on the height of the tile it is computed in (by the batch and the range: 16 to 128 rows), a sine past its reduction among them."""
    from vox_serve_b200.tokenizer import _cl

    T, g = rows + 5, torch.Generator(device="cuda").manual_seed(rows + C)
    x, w = torch.randn(80, T, C, generator=g, device="cuda"), torch.randn(7, C, generator=g, device="cuda")
    x[::3, rows // 2, 5] = 3e5
    b, *a = (torch.rand(C, generator=g, device="cuda") + 0.5 for _ in range(3))
    a = [torch.cat((v, 1 / (v + 1e-9))) for v in a]

    def result(x, lo, hi):
        n = x.numel()
        y = _cl.depthwise7(_cl.Act(x.reshape(-1).clone(), x.shape[0], T, C), w, b, *a, dil, lo, hi, parts=parts).buf
        bits = y[:n].view(torch.int32).view(-1, T, C)[:, lo:hi].clone()
        return torch.cat((bits, y[n:].view(torch.uint8)[:n // 32].view(-1, T, C // 32)[:, lo:hi].int()), 2) if parts else bits

    whole = result(x, 3, 3 + rows)
    for n in (1, 3, 9, 20, 40):
        assert torch.equal(result(x[:n], 3, 3 + rows), whole[:n]), n
    for lo in {3, 3 + rows // 2, 2 + rows}:
        assert torch.equal(result(x[:2], lo, lo + 1), whole[:2, lo - 3: lo - 2]), lo
    if not parts:
        v = x[:4].double().transpose(1, 2)
        snake = lambda v, a: v + torch.sin((v.float() * a[:C, None]).double()) ** 2 / (a[:C].double()[:, None] + 1e-9)  # noqa: E731
        v = torch.nn.functional.conv1d(snake(v, a[0]), w.t().double()[:, None], b.double(), dilation=dil, padding=3 * dil, groups=C)
        ref = snake(v, a[1]).transpose(1, 2)[:, 3:3 + rows]
        bad = ref.abs() > 1e4                                                    # (the second sine's argument has rounded by more than its period there)
        _close(torch.where(bad, 0, whole[:4].view(torch.float32)), torch.where(bad, 0, ref), 5e-6)


@pytest.mark.parametrize("B,T,C,dil,lo,hi", [(1, 1, 64, 1, 0, 1), (2, 127, 64, 3, 0, 127), (3, 253, 128, 9, 7, 251), (1, 300, 256, 1, 0, 300), (40, 130, 128, 9, 0, 130),
                                             (2, 65, 192, 3, 0, 65), (1, 40, 1024, 1, 0, 40), (2, 1000, 64, 9, 111, 999), (1, 500, 64, 64, 0, 500), (5, 33, 320, 5, 1, 32)])
@pytest.mark.parametrize("last", [False, True])
@pytest.mark.parametrize("odd", [False, True])
def test_channels_last_residual_unit(B, T, C, dil, lo, hi, last, odd):
    """A unit in one launch is the same bits as its depthwise and its 1x1 convolution, also where parts cannot hold a value; and an entry's do not depend on its batch."""
    from vox_serve_b200 import _lib
    from vox_serve_b200.tokenizer import _cl

    g = torch.Generator(device="cuda").manual_seed(B * T + C + dil)
    rnd = lambda *s, std=1.0: torch.randn(*s, generator=g, device="cuda") * std          # noqa: E731
    x, dw, db, w, b = rnd(B, T, C), rnd(7, C, std=7 ** -0.5), rnd(C, std=0.05), _cl.pack(rnd(C, C, std=C ** -0.5)), rnd(C, std=0.05)
    a = [torch.cat((v, 1.0 / (v + 1e-9))) for v in (0.5 + torch.rand(C, generator=g, device="cuda") for _ in range(3))]
    if odd:
        db.zero_()
        x[0, T // 2, 3] = 1e6                      # out of the parts' range, and past what the sine reduces
        x[-1, T // 3] *= 1e-9
        x[0, T // 4] = 0.0
        x[-1, T - 1, C - 1] = float("nan")

    def fused(v):
        X = _cl.Act(v.contiguous().view(-1), v.shape[0], T, C)
        return X, _cl.dw_unit(X, dw, db, a[0], a[1], w, b, dil, lo, hi, a[2] if last else None, "parts" if last else "f32")

    def bits(y):
        n = y.B * T * C
        codes = y.buf.view(torch.uint8)[4 * n:4 * n + n // 32].view(y.B, T, -1)[:, lo:hi] if y.parts else torch.zeros(1, device="cuda")
        return y.buf[:n].view(torch.int32).view(y.B, T, C)[:, lo:hi], codes

    X, got = fused(x)
    h = _cl.depthwise7(X, dw, db, a[0], a[1], dil, lo, hi, parts=True)
    want = _cl.conv(h, w, C, b, epi="resid", resid=X, act="snake" if last else None, alpha=a[2] if last else None, lo=lo, hi=hi, out="parts" if last else "f32")
    for p, q in zip(bits(got), bits(want)):
        assert torch.equal(p, q)
    for p, q in zip(bits(fused(x[-1:])[1]), bits(got)):
        assert torch.equal(p, q[-1:] if p.dim() == 3 else q)
    assert _lib.load().vb_cl_timeouts() == 0


@pytest.mark.parametrize("B,T", [(1, 1), (3, 4), (2, 123), (2, 124), (1, 125), (3, 249), (2, 1000), (300, 130)])
@pytest.mark.parametrize("kind", ["plain", "one", "quiet", "mixed", "nan", "hidden"])
def test_channels_last_tail(B, T, kind):
    """The last unit of Mimi and its convolution to one channel in one launch against 64 bits, also where parts cannot hold a value; and an entry alone."""
    from vox_serve_b200 import _lib
    from vox_serve_b200.tokenizer import _cl

    g = torch.Generator(device="cuda").manual_seed(7 * B + T)
    rnd = lambda *s, std=1.0: torch.randn(*s, generator=g, device="cuda") * std          # noqa: E731
    w1, b1, w3, b3 = rnd(32, 64, 3, std=192 ** -0.5), rnd(32, std=0.05), rnd(64, 32, std=0.5 * 32 ** -0.5), rnd(64, std=0.05)
    wl, bl, x = rnd(1, 64, 3, std=0.5 * 192 ** -0.5), rnd(1, std=0.01), rnd(B, T, 64)
    if kind == "one":
        x[0, T // 2, 3] = 1e6
    elif kind == "quiet":
        x *= 1e-9
    elif kind == "mixed":
        x[:, ::3] *= 1e4
        x[:, 1::3] *= 1e-7
    elif kind == "nan":
        x[-1, T // 2, 63] = float("nan")
    elif kind == "hidden":                         # parts hold the inputs, not what is made of them
        w1, b1 = w1 * 3e4, b1 * 0
        w1[::2] *= 1e-9
    p1, p3, wf = _cl.pack_conv(w1.reshape(32, -1), 64, 3), _cl.pack(w3), wl.reshape(1, -1).contiguous()
    run = lambda v: _cl.res_tail(_cl.Act(v.contiguous().view(-1), v.shape[0], T, 64), p1, b1, p3, b3, wf, bl)          # noqa: E731
    got = run(x)
    elu = lambda v: v.where(v > 0, torch.expm1(v))          # noqa: E731

    def taps(v, w):                                # a product per tap (the library's convolution spreads a NaN further than its taps)
        k = w.shape[2]
        v = torch.cat((v.new_zeros(B, k - 1, v.shape[2]), v), 1)
        return sum(v[:, j:j + T] @ w[:, :, j].T for j in range(k))

    d, e = x.double(), [v.double() for v in (w1, b1, w3[:, :, None], b3, wl, bl)]
    h = taps(elu(d), e[0]) + e[1]
    want = (taps(elu(d + taps(elu(h), e[2]) + e[3]), e[4]) + e[5]).transpose(1, 2)
    assert torch.equal(got.isnan(), want.isnan())
    ok = want.isfinite()
    # both factors to 2^-22, sums of 192 in 32 bits: 1.4e-7 measured, as with a launch a convolution
    assert float((got.double() - want)[ok].norm()) <= 5e-7 * float(want[ok].norm())
    assert torch.equal(run(x[-1:])[0].view(torch.int32), got[-1].view(torch.int32))
    assert _lib.load().vb_cl_timeouts() == 0


def _us(f):
    times = []
    for _ in range(6):
        a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
        a.record()
        for _ in range(4):
            f()
        b.record()
        b.synchronize()
        times.append(a.elapsed_time(b) * 250)
    return min(times)


@pytest.mark.parametrize("kind", ["plain", "zero", "one a tile", "silence", "quiet", "loud"])
def test_channels_last_residual_unit_is_no_slower_than_its_convolutions(kind):
    """One launch against the depthwise and the 1x1 convolution, whatever its inputs are (0.7 to 1.05 of their time; once 1.9 with loud values, 3 with zeros)."""
    from vox_serve_b200.tokenizer import _cl

    B, T, C, dil = 32, 6000, 64, 9
    g = torch.Generator(device="cuda").manual_seed(1)
    rnd = lambda *s, std=1.0: torch.randn(*s, generator=g, device="cuda") * std          # noqa: E731
    x, dw, w, b = rnd(B, T, C), rnd(7, C, std=7 ** -0.5), _cl.pack(rnd(C, C, std=C ** -0.5)), rnd(C, std=0.05)
    db = torch.zeros(C, device="cuda") if kind in ("zero", "quiet", "silence") else rnd(C, std=0.05)
    a = [torch.cat((v, 1.0 / (v + 1e-9))) for v in (0.5 + torch.rand(C, generator=g, device="cuda") for _ in range(2))]
    if kind == "one a tile":
        x[:, 50::124, 3] = 1e6
    elif kind == "silence":
        x[:, T // 2:T // 2 + 240] *= 1e-9
    elif kind != "plain":
        x *= {"zero": 0.0, "quiet": 1e-9, "loud": 1e6}[kind]
    X = _cl.Act(x.view(-1), B, T, C)

    def launches():
        return _cl.conv(_cl.depthwise7(X, dw, db, *a, dil, 0, T, parts=True), w, C, b, epi="resid", resid=X)

    one, two = _us(lambda: _cl.dw_unit(X, dw, db, *a, w, b, dil, 0, T)), _us(launches)
    assert one <= 1.5 * two, (one, two)


def _tail_weights(g):
    """weights of the end of Mimi's decoder, as it keeps them"""
    from vox_serve_b200.tokenizer import _cl

    rnd = lambda *s, std=1.0: torch.randn(*s, generator=g, device="cuda") * std          # noqa: E731
    w1, b1, w3, b3 = rnd(32, 64, 3, std=192 ** -0.5), rnd(32, std=0.05), rnd(64, 32, std=0.5 * 32 ** -0.5), rnd(64, std=0.05)
    return _cl.pack_conv(w1.reshape(32, -1), 64, 3), b1, _cl.pack(w3), b3, rnd(1, 192, std=0.5 * 192 ** -0.5), rnd(1, std=0.01)


@pytest.mark.parametrize("where", [0, 60, 122, 130, 379])
def test_channels_last_tail_beside_a_loud_value(where):
    """Positions that a loud value is not part of keep their bits, in its tile and in its warp."""
    from vox_serve_b200.tokenizer import _cl

    g, T = torch.Generator(device="cuda").manual_seed(where), 380
    w, x = _tail_weights(g), torch.randn(2, T, 64, generator=g, device="cuda")
    run = lambda: _cl.res_tail(_cl.Act(x.clone().view(-1), 2, T, 64), *w).view(2, T)     # noqa: E731
    plain = run()
    x[1, where, 7] = 1e6
    got = run()
    far = torch.ones(2, T, dtype=torch.bool, device="cuda")
    far[1, where:where + 5] = False              # (two taps, two taps)
    assert torch.equal(got[far], plain[far]) and not torch.equal(got[~far], plain[~far])


@pytest.mark.parametrize("kind", ["plain", "one", "one a tile", "silence", "quiet", "loud"])
def test_channels_last_tail_is_no_slower_than_its_convolutions(kind):
    """One launch against a launch a convolution, whatever its inputs are: what parts cannot hold is a warp's work and not a lane's (0.3 to 0.6 of their time; once 14 times)."""
    from vox_serve_b200.tokenizer import _cl

    B, T = 8, 9600
    g = torch.Generator(device="cuda").manual_seed(1)
    (w1, b1, w3, b3, wl, bl), x = _tail_weights(g), torch.randn(B, T, 64, generator=g, device="cuda")
    if kind == "one":
        x[0, T // 2, 3] = 1e6
    elif kind == "one a tile":
        x[:, 50::124, 3] = 1e6
    elif kind == "silence":
        x[:, T // 2:T // 2 + 240] *= 1e-9
    elif kind != "plain":
        x *= 1e-9 if kind == "quiet" else 1e5
    X = _cl.Act(x.view(-1), B, T, 64)
    xp = _cl.conv(X, _cl.pack(torch.eye(64, device="cuda")), 64, act="elu", out="parts")

    def launches():
        h = _cl.conv(xp, w1, 32, b1, ksize=3, act="elu", out="parts")
        return _cl.last_conv(_cl.conv(h, w3, 64, b3, epi="resid", resid=X, act="elu"), wl, bl, 3, 2, 0, T, tanh=False)

    one, three = _us(lambda: _cl.res_tail(X, w1, b1, w3, b3, wl, bl)), _us(launches)
    assert one <= 1.5 * three, (one, three)


@pytest.mark.parametrize("B,T,C,ksize,left,lo,hi", [(1, 1, 64, 3, 2, 0, 1), (2, 129, 96, 3, 2, 0, 129), (3, 40, 4, 3, 0, 5, 38), (1, 300, 256, 7, 3, 1, 300), (2, 17, 68, 5, 4, 0, 17),
                                                   (1, 130, 128, 16, 15, 0, 130), (2, 16, 32, 1, 0, 0, 16)])
def test_channels_last_one_output_channel(B, T, C, ksize, left, lo, hi):
    """Runs of sixteen positions with and without rows before and behind the sequence; a position's sum is the same wherever it lies."""
    from vox_serve_b200.tokenizer import _cl

    g = torch.Generator(device="cuda").manual_seed(T + C)
    x, w, b = (torch.randn(*n, generator=g, device="cuda") for n in ((B, T, C), (C, ksize), (1,)))
    act = _cl.Act(x.reshape(-1).clone(), B, T, C)
    y = _cl.last_conv(act, w, b, ksize, left, lo, hi, tanh=False)
    ref = torch.nn.functional.conv1d(torch.nn.functional.pad(x.double().transpose(1, 2), (left, ksize - 1)), w.double()[None], b.double())[..., lo:hi]
    _close(y, ref, 2e-6)                       # chains of at most 4 * ksize * C / 64 roundings and four additions
    if hi - lo > 3:
        assert torch.equal(_cl.last_conv(act, w, b, ksize, left, lo + 3, hi, tanh=False), y[..., 3:])


@pytest.mark.parametrize("B,T,H,D,parts", [(1, 1, 1, 4, False), (2, 20, 8, 64, True), (1, 33, 2, 32, True), (2, 64, 3, 128, True), (1, 64, 1, 256, True), (3, 31, 2, 36, False), (1, 9, 2, 68, False)])
def test_vocoder_chunk_attention_and_norm(B, T, H, D, parts):
    from vox_serve_b200._lib import call
    from vox_serve_b200.tokenizer import _cl

    C, period = H * D, 1e4
    g = torch.Generator(device="cuda").manual_seed(T + D)
    buf = torch.randn(B * T * 3 * C + 2, generator=g, device="cuda")
    for at in (0, 2):                          # rows on 16- and on 8-byte boundaries
        qkv = buf[at:at + B * T * 3 * C].view(B, T, 3, H, D)
        out = _cl.Act.empty(B, T, C, "cuda", parts)
        call("vb_cl_chunk_attention_parts", out.ptr, out.codes, qkv.data_ptr(), B, C, H, T, period, 0)
        torch.cuda.synchronize()
        got = _cl.conv(out, _cl.pack(torch.eye(C, device="cuda")), C).tensor() if parts else out.tensor()
        angle = torch.arange(T, device="cuda")[:, None].double() * torch.exp(torch.arange(D // 2, device="cuda").double() * (-math.log(period) * 2 / D))
        rot = torch.polar(torch.ones_like(angle), angle)
        turn = lambda t: torch.view_as_real(torch.view_as_complex(t.double().reshape(B, T, H, D // 2, 2).contiguous()) * rot[:, None]).flatten(-2)   # noqa: E731
        q, k, v = turn(qkv[:, :, 0]), turn(qkv[:, :, 1]), qkv[:, :, 2].double()
        s = torch.einsum("bqhd,bkhd->bhqk", q, k) * D ** -0.5
        s = s.masked_fill(torch.ones(T, T, device="cuda").triu(1).bool(), -math.inf).softmax(-1)
        _close(got, torch.einsum("bhqk,bkhd->bqhd", s, v).reshape(B, T, C), 5e-6)       # scores of a few units: their roundings reach the weights
    x, w, b = torch.randn(B * T, C, generator=g, device="cuda") + 3, *torch.randn(2, C, generator=g, device="cuda")
    if C <= 1024:
        y = _cl.Act.empty(B, T, C, "cuda")
        call("vb_cl_layernorm_parts", y.ptr, None, x.data_ptr(), w.contiguous().data_ptr(), b.contiguous().data_ptr(), B * T, C, 1e-5, 0)
        torch.cuda.synchronize()
        _close(y.tensor().reshape(B * T, C), torch.nn.functional.layer_norm(x.double(), (C,), w.double(), b.double(), 1e-5), 2e-6)
    if T > 2:                                  # a value that is not a number stays out of the positions before it
        buf[2 * C * 3 + 2 * C] = math.nan
        out = _cl.Act.empty(B, T, C, "cuda")
        call("vb_cl_chunk_attention_parts", out.ptr, None, buf.data_ptr(), B, C, H, T, period, 0)
        torch.cuda.synchronize()
        assert torch.isfinite(out.tensor()[0, :2]).all() and torch.isnan(out.tensor()[0, 2:, 0]).all()


# prompt rows of window attention on tcgen05: head sizes, heads per key head (rows per tile), page sizes down to one 8-token group, row
# tiles of one row and of 64, windows and chunks that start inside key tiles, kept tokens near and far, sinks, both gates, fp32 output
@pytest.mark.parametrize("D,H,G,page,new,old,window,chunk,keep,sink,gate,share,f32", [
    (128, 4, 1, 64, [1, 64, 65], [0, 0, 0], 0, 0, 0, False, None, 1, False), (64, 6, 2, 8, [130], [0], 0, 0, 0, True, "head", 1, False),
    (128, 3, 3, 16, [70, 3], [200, 61], 50, 0, 0, False, "value", 1, True), (64, 16, 1, 32, [100], [300], 64, 0, 5, True, None, 1, False),
    (128, 8, 2, 64, [129], [500], 130, 0, 70, True, "head", 1, False), (64, 4, 4, 64, [200], [10], 0, 96, 0, False, None, 2, False),
    (128, 130, 10, 64, [33], [31], 0, 0, 0, False, None, 1, False), (64, 200, 2, 24, [5], [64], 3, 0, 2, False, None, 1, False)])
def test_window_attention_prompt_rows(ops, D, H, G, page, new, old, window, chunk, keep, sink, gate, share, f32):
    from vox_serve_b200 import _lib

    g = torch.Generator(device="cuda").manual_seed(H * D + page)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")                 # noqa: E731
    n, T, Gv = [a + b for a, b in zip(new, old)], sum(new), G // share
    pages = [(x + page - 1) // page for x in n]
    ip = np.concatenate([[0], np.cumsum(pages)]).tolist()
    idx = np.random.RandomState(T).permutation(ip[-1]).tolist()
    # what no position of a request has written is not a number: nothing of it may reach a result
    kc, vc = (torch.full((ip[-1], page, h, D), float("nan"), device="cuda").bfloat16() for h in (G, Gv))
    q, snk = rnd(T, H, D).bfloat16(), rnd(H) if sink else None
    gt = rnd(T, H if gate == "head" else H * D) if gate else None
    ref, at, treq, trow, pos = [], 0, [], [], []
    for b, L in enumerate(n):
        k, v = rnd(L, G, D).bfloat16(), rnd(L, Gv, D).bfloat16()
        tok = torch.arange(L, device="cuda")
        pg = torch.tensor(idx[ip[b]:ip[b + 1]], device="cuda")[tok // page]
        kc[pg, tok % page], vc[pg, tok % page] = k, v
        i, j = torch.arange(old[b], L, device="cuda")[:, None], tok[None]
        lo = torch.zeros_like(i) if not window else (i - window + 1).clamp(min=0)
        lo = torch.maximum(lo, i - i % chunk) if chunk else lo
        seen = (j <= i) & ((j >= lo) | (j < keep))
        for h in range(H):
            kg = h // (H // G)
            s = (q[at:at + new[b], h].double() @ k[:, kg].double().T * D ** -0.5).masked_fill(~seen, -float("inf"))
            if sink:
                s = torch.cat((s, snk[h].double().expand(new[b], 1)), 1)
            ref.append((torch.softmax(s, -1)[:, :L] @ v[:, kg // share].double(), at, h))
        for r in range(0, new[b], 64):
            treq.append(b)
            trow.append(at + r)
        pos += list(range(old[b], L))
        at += new[b]
    want = torch.empty(T, H, D, dtype=torch.float64, device="cuda")
    for o, t0, h in ref:
        want[t0:t0 + o.shape[0], h] = o
    if gate:
        want = want * torch.sigmoid(gt.double().view(T, H, -1))
    out = torch.full((T, H * D), float("nan"), device="cuda", dtype=torch.float32 if f32 else torch.bfloat16)
    ops.window_attn(q.view(T, H * D), kc, vc, out, gt, None, _i32(pos), _i32(ip), _i32(idx), T, H, G, D, D, window, D ** -0.5,
                    tiles=(_i32([0] + np.cumsum(new).tolist()), _i32(treq), _i32(trow), len(treq)), chunk=chunk, v_share=share, sink=snk,
                    keep_first=keep, head_gate=gate == "head")
    _close(out.view(T, H, D), want, 2 ** -8)         # probabilities and the output rounded to bf16
    assert _lib.load().vb_window_attn_tc_timeouts() == 0


# keys between the kept tokens and the first one that a row tile sees: inside a key tile, over several, inside the tile of the kept tokens,
# from a chunk's start, none at all; pages larger and smaller than what they cover
@pytest.mark.parametrize("D,H,G,page,new,old,window,chunk,keep", [
    (128, 4, 2, 64, 20, 500, 100, 0, 0), (64, 4, 4, 8, 60, 300, 50, 0, 5), (128, 8, 2, 16, 32, 200, 30, 0, 70), (64, 2, 1, 32, 10, 100, 0, 96, 0),
    (128, 2, 2, 16, 40, 80, 45, 0, 20), (128, 2, 2, 16, 40, 60, 45, 0, 20), (64, 4, 1, 24, 3, 1000, 1, 0, 65)])
def test_window_attention_unseen_keys(ops, D, H, G, page, new, old, window, chunk, keep):
    """Nothing of the keys that no row sees reaches a result, and their pages need not be the request's."""
    g = torch.Generator(device="cuda").manual_seed(old)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()      # noqa: E731
    L = old + new
    first = lambda i: max(i - window + 1 if window else 0, i - i % chunk if chunk else 0, 0)     # noqa: E731
    hole = range(min(keep, first(old)), first(old))
    n = (L + page - 1) // page
    idx = np.random.RandomState(L).permutation(n).tolist()
    kc, vc = (torch.full((n + 1, page, G, D), float("nan"), device="cuda").bfloat16() for _ in range(2))
    q, k, v = rnd(new, H, D), rnd(L, G, D), rnd(L, G, D)
    for j in range(L):
        if j not in hole:
            kc[idx[j // page], j % page], vc[idx[j // page], j % page] = k[j], v[j]
    table = [n if set(range(i * page, (i + 1) * page)) <= set(hole) else idx[i] for i in range(n)]
    i, j = torch.arange(old, L, device="cuda")[:, None], torch.arange(L, device="cuda")[None]
    lo = torch.tensor([first(a) for a in range(old, L)], device="cuda")[:, None]
    seen = (j <= i) & ((j >= lo) | (j < keep))
    kk, vv = (x.double().repeat_interleave(H // G, 1) for x in (k, v))
    s = torch.einsum("qhd,khd->hqk", q.double(), kk) * D ** -0.5
    want = torch.einsum("hqk,khd->qhd", torch.softmax(s.masked_fill(~seen, -float("inf")), -1), vv)
    out = torch.full((new, H * D), float("nan"), device="cuda").bfloat16()
    ops.window_attn(q.view(new, H * D), kc, vc, out, None, None, _i32(list(range(old, L))), _i32([0, n]), _i32(table), new, H, G, D, D, window,
                    D ** -0.5, tiles=(_i32([0, new]), _i32([0]), _i32([0]), 1), chunk=chunk, keep_first=keep)
    _close(out.view(new, H, D), want, 2 ** -8)


# boxes of 8, 16, 32 and 64 tokens and pages that no box divides (copied row by row); requests that end on a key tile, one before and one
# behind it; rows that see one tile, two, several; heads per key head from one to a whole row tile
@pytest.mark.parametrize("page", [8, 24, 16, 32, 96, 64, 192, 1, 5, 20, 66])
@pytest.mark.parametrize("D,H,G,kv,new", [(128, 6, 2, [63, 64, 65], [63, 1, 65]), (64, 4, 4, [127, 129, 300], [127, 70, 40]), (128, 64, 1, [1, 130], [1, 3])])
def test_paged_prompt_attention_pages(ops, page, D, H, G, kv, new):
    from vox_serve_b200 import _lib

    g = torch.Generator(device="cuda").manual_seed(page)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()      # noqa: E731
    pages = [(x + page - 1) // page for x in kv]
    ip = np.concatenate([[0], np.cumsum(pages)]).tolist()
    idx = (np.random.RandomState(page).permutation(ip[-1]) + 1).tolist()
    T, pad, base = sum(new), 3, 2
    cache = torch.full((base + ip[-1] + 1, 2, page, G, D), float("nan"), device="cuda").bfloat16()       # what no request has written
    q, want, at = rnd(T + pad, H, D), [], 0
    for b, L in enumerate(kv):
        k, v, tok = rnd(L, G, D), rnd(L, G, D), torch.arange(L, device="cuda")
        pg = torch.tensor(idx[ip[b]:ip[b + 1]], device="cuda")[tok // page] + base
        cache[pg, 0, tok % page], cache[pg, 1, tok % page] = k, v
        s = torch.einsum("qhd,khd->hqk", q[at:at + new[b]].double(), k.double().repeat_interleave(H // G, 1)) * D ** -0.5
        s = s.masked_fill(tok[None] > torch.arange(L - new[b], L, device="cuda")[:, None], -float("inf"))
        want.append(torch.einsum("hqk,khd->qhd", torch.softmax(s, -1), v.double().repeat_interleave(H // G, 1)))
        at += new[b]
    plan = ops.RowPlan(T + pad, "cuda")
    chunk = page
    ops.plan_rows(plan, _i32([0] + np.cumsum(new).tolist()), _i32(ip), _i32(idx), _i32([(x - 1) % page + 1 for x in kv]), len(kv), T + pad, page, chunk)
    out = torch.full((T + pad, H, D), 7.0, device="cuda").bfloat16()
    ops.paged_attn(q, cache, base, plan, T + pad, G, page, chunk, None, out=out, prefill_tiles="tc")
    _close(out[:T], torch.cat(want), 2 ** -8)        # probabilities and the output rounded to bf16
    assert (out[T:] == 0).all()
    assert _lib.load().vb_prefill_attn_tc_timeouts() == 0


# rows on several key tiles, one key before and behind the end of a key tile; a last key tile of one key, with rows of the tile that see nothing
# of it; boxes and rows of cp.async; both layouts of the result
@pytest.mark.parametrize("page,tiled", [(64, True), (16, False), (20, False)])
@pytest.mark.parametrize("D,H,G,kv,new", [(128, 6, 2, [320, 321, 384, 385], [1, 64, 100, 43]), (64, 4, 4, [449, 1000, 64], [449, 3, 2])])
def test_paged_prompt_attention_several_tiles(ops, page, tiled, D, H, G, kv, new):
    from vox_serve_b200 import _lib

    g = torch.Generator(device="cuda").manual_seed(page + D)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()      # noqa: E731
    pages = [(x + page - 1) // page for x in kv]
    ip = np.concatenate([[0], np.cumsum(pages)]).tolist()
    T, q = sum(new), rnd(sum(new), H, D)
    cache = torch.full((ip[-1], 2, page, G, D), float("nan"), device="cuda").bfloat16()
    want, at = [], 0
    for b, L in enumerate(kv):
        k, v, tok = rnd(L, G, D), rnd(L, G, D), torch.arange(L, device="cuda")
        cache[ip[b] + tok // page, 0, tok % page], cache[ip[b] + tok // page, 1, tok % page] = k, v
        s = torch.einsum("qhd,khd->hqk", q[at:at + new[b]].double(), k.double().repeat_interleave(H // G, 1)) * D ** -0.5
        s = s.masked_fill(tok[None] > torch.arange(L - new[b], L, device="cuda")[:, None], -float("inf"))
        want.append(torch.einsum("hqk,khd->qhd", torch.softmax(s, -1), v.double().repeat_interleave(H // G, 1)))
        at += new[b]
    plan = ops.RowPlan(T, "cuda")
    ops.plan_rows(plan, _i32([0] + np.cumsum(new).tolist()), _i32(ip), _i32(list(range(ip[-1]))), _i32([(x - 1) % page + 1 for x in kv]), len(kv), T,
                  page, page)
    out = ops.TiledAct(T, H * D, "cuda") if tiled else None
    out = ops.paged_attn(q, cache, 0, plan, T, G, page, page, None, out=out, prefill_tiles="tc")
    got = out.to_rows().view(T, H, D) if tiled else out
    _close(got, torch.cat(want), 2 ** -8)            # probabilities and the output rounded to bf16
    assert _lib.load().vb_prefill_attn_tc_timeouts() == 0


@pytest.mark.parametrize("D,H,G,kv,new,at", [(128, 6, 2, 400, 400, 1), (64, 4, 4, 700, 100, 0), (128, 8, 1, 1500, 37, 2)])
def test_paged_prompt_attention_alone_and_in_a_step(ops, D, H, G, kv, new, at):
    """A request's rows are the same bits alone, beside other prompts, and in portions; through the operator shim too."""
    from vox_serve_b200.flashinfer_utils import FlashInferPrefillWrapper

    page, g = 64, torch.Generator(device="cuda").manual_seed(kv)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()      # noqa: E731
    pages = lambda n: (n + page - 1) // page                                     # noqa: E731
    others = [(900, 900), (1030, 700), (64, 64)]                                 # (cached with the new rows, new)
    reqs = others[:at] + [(kv, new)] + others[at:]
    first = np.concatenate([[0], np.cumsum([pages(n) for n, _ in reqs])]).tolist()
    cache, q = rnd(first[-1], 2, page, G, D), [rnd(r, H, D) for _, r in reqs]

    def run(chosen, shim=False):
        """chosen: (request, its rows from, to) of the step"""
        lens = [reqs[i][0] - reqs[i][1] + b for i, _, b in chosen]
        idx = [first[i] + j for (i, _, _), n in zip(chosen, lens) for j in range(pages(n))]
        qo, ip = ([0] + np.cumsum(v).tolist() for v in ([b - a for _, a, b in chosen], [pages(n) for n in lens]))
        last, rows = [(n - 1) % page + 1 for n in lens], torch.cat([q[i][a:b] for i, a, b in chosen])
        if shim:
            w = FlashInferPrefillWrapper(attn_buffer=None, n_qo_head=H, n_kv_head=G, n_state=H * D, page_size=page, device="cuda", max_seq_len=4096)
            w.plan(*(torch.tensor(v, dtype=torch.int32) for v in (qo, ip, idx, last)))
            out = w.run(rows, cache).view(-1, H, D)
        else:
            plan = ops.RowPlan(qo[-1], "cuda")
            ops.plan_rows(plan, _i32(qo), _i32(ip), _i32(idx), _i32(last), len(chosen), qo[-1], page, page)
            out = ops.paged_attn(rows, cache, 0, plan, qo[-1], G, page, page, None, prefill_tiles="tc")
        n = [i for i, _, _ in chosen].index(at)
        return out[qo[n]:qo[n + 1]]

    step = [(i, 0, r) for i, (_, r) in enumerate(reqs)]
    want = run([(at, 0, new)])
    assert torch.equal(run(step), want)
    cut = new // 3
    assert torch.equal(torch.cat((run([(at, 0, cut)]), run(step[:at] + [(at, cut, new)] + step[at + 1:]))), want)
    if new >= 100:                                       # (fewer rows alone take the row kernel)
        assert torch.equal(run([(at, 0, new)], True), run(step, True))


@pytest.mark.parametrize("n,old,window,keep", [(500, 0, 0, 0), (640, 100, 300, 4)])
def test_window_attention_alone_and_in_a_step(ops, n, old, window, keep):
    """A prompt's rows are the same bits alone and beside other prompts."""
    D, H, G, page = 128, 16, 4, 64
    g = torch.Generator(device="cuda").manual_seed(n)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()      # noqa: E731
    reqs = [(1000, 0), (n, old), (900, 0)]
    pages = [(r + o + page - 1) // page for r, o in reqs]
    first = np.concatenate([[0], np.cumsum(pages)]).tolist()
    q, kc, vc = [rnd(r, H * D) for r, _ in reqs], rnd(first[-1], page, G, D), rnd(first[-1], page, G, D)

    def run(chosen):
        T, qo, treq, trow, pos, idx, ip = 0, [0], [], [], [], [], [0]
        for k, i in enumerate(chosen):
            r, o = reqs[i]
            treq += [k] * ((r + 63) // 64)
            trow += list(range(T, T + r, 64))
            pos += list(range(o, o + r))
            idx += list(range(first[i], first[i + 1]))
            T += r
            qo.append(T)
            ip.append(len(idx))
        out = torch.empty(T, H * D, device="cuda").bfloat16()
        ops.window_attn(torch.cat([q[i] for i in chosen]), kc, vc, out, None, None, _i32(pos), _i32(ip), _i32(idx), T, H, G, D, D, window, D ** -0.5,
                        tiles=(_i32(qo), _i32(treq), _i32(trow), len(treq)), keep_first=keep)
        k = chosen.index(1)
        return out[qo[k]:qo[k + 1]]

    assert torch.equal(run([0, 1, 2]), run([1]))

def test_a_plan_of_pinned_tables_inside_a_graph(ops):
    """Pinned tables are copied from where they lie: a plan can be captured, and every replay reads them again."""
    from vox_serve_b200.flashinfer_utils import FlashInferDecodeWrapper, FlashInferPrefillWrapper

    D, H, G, page = 128, 6, 2, 16
    g = torch.Generator(device="cuda").manual_seed(5)
    cache = torch.randn(24, 2, page, G, D, generator=g, device="cuda").bfloat16()
    pin = lambda v: torch.tensor(v, dtype=torch.int32).pin_memory()              # noqa: E731
    for cls, new in ((FlashInferPrefillWrapper, [40, 23]), (FlashInferDecodeWrapper, [1, 1])):
        q = torch.randn(sum(new), H, D, generator=g, device="cuda").bfloat16()
        tables = [pin(v) for v in ([0, new[0], sum(new)], [0, 4, 9], list(range(9)), [9, 3])][0 if len(q) > 2 else 1:]
        make = lambda: cls(attn_buffer=None, n_qo_head=H, n_kv_head=G, n_state=H * D, page_size=page, device="cuda")     # noqa: E731
        w = make()
        w.plan(*tables)
        w.run(q, cache)
        torch.cuda.synchronize()
        graph, s = torch.cuda.CUDAGraph(), torch.cuda.Stream()
        with torch.cuda.graph(graph, stream=s):
            w.plan(*tables)
            out = w.run(q, cache)
        for idx, last in (([3, 20, 5, 11, 0, 7, 23, 2, 9], [16, 5]), ([8, 7, 6, 5, 4, 3, 2, 1, 0], [9, 16])):
            tables[-2].copy_(torch.tensor(idx))
            tables[-1].copy_(torch.tensor(last))
            graph.replay()
            torch.cuda.synchronize()
            ref = make()
            ref.plan(*(t.clone() for t in tables))
            assert torch.equal(out, ref.run(q, cache))


@pytest.mark.parametrize("H", [128, 129, 200])
def test_paged_prompt_attention_many_heads_per_key_head(ops, H):
    """More query heads on one key head than a tcgen05 row tile has rows: an automatic plan runs all the same."""
    D, page, L = 64, 16, 40
    g = torch.Generator(device="cuda").manual_seed(H)
    q, cache = (torch.randn(*s, generator=g, device="cuda").bfloat16() for s in ((L, H, D), (3, 2, page, 1, D)))
    plan = ops.RowPlan(L, "cuda")
    ops.plan_rows(plan, _i32([0, L]), _i32([0, 3]), _i32([0, 1, 2]), _i32([8]), 1, L, page, page)
    out = ops.paged_attn(q, cache, 0, plan, L, 1, page, page, None)
    k, v = (cache[:, i, :, 0].reshape(-1, D)[:L].double() for i in (0, 1))
    s = torch.einsum("qhd,kd->hqk", q.double(), k) * D ** -0.5
    s = s.masked_fill(torch.ones(L, L, device="cuda").triu(1).bool(), -float("inf"))
    _close(out, torch.einsum("hqk,kd->qhd", torch.softmax(s, -1), v), 2 ** -8)


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("width", [1.0, 3.0])
def test_prompt_attention_probabilities(ops, D, width):
    """The attention core of prompt rows with fp32 output: probabilities are two bf16 terms (2^-17 together), their sum and the products
    32-bit, whatever the reference of the exponents (one bf16 term against the exact maximum: 2^-10 or so)."""
    H, new, L, page = 4, 256, 1000, 64
    g = torch.Generator(device="cuda").manual_seed(D)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")                 # noqa: E731
    n = (L + page - 1) // page
    q, k, v = (rnd(new, H, D) * width).bfloat16(), rnd(n * page, H, D).bfloat16(), rnd(n * page, H, D).bfloat16()
    out = torch.full((new, H * D), float("nan"), device="cuda")
    ops.window_attn(q.view(new, H * D), k.view(n, page, H, D), v.view(n, page, H, D), out, None, None, _i32(list(range(L - new, L))), _i32([0, n]),
                    _i32(list(range(n))), new, H, H, D, D, 0, D ** -0.5, tiles=(_i32([0, new]), _i32(list([0] * 4)), _i32([0, 64, 128, 192]), 4))
    s = torch.einsum("qhd,khd->hqk", q.double(), k[:L].double()) * D ** -0.5
    s = s.masked_fill(torch.arange(L, device="cuda")[None] > torch.arange(L - new, L, device="cuda")[:, None], -float("inf"))
    vd = v[:L].double().transpose(0, 1)
    want = torch.softmax(s, -1) @ vd
    err = ((out.view(new, H, D).transpose(0, 1).double() - want).norm() / want.norm()).item()
    assert err <= 2.0 ** -15, err


@pytest.mark.parametrize("T,N,S,resid,tiled,hidden", [
    (513, 8, 1, True, False, True), (514, 2048, 3, True, True, True), (600, 3072, 1, False, True, False), (515, 4096, 2, True, False, True),
    (516, 1032, 9, True, False, True), (1024, 264, 1, True, False, False),
])
def test_reduce_residual_rmsnorm_many_rows(ops, T, N, S, resid, tiled, hidden):
    """A step of more than 512 rows against the same rows in steps of at most 148, which take the kernel of few rows."""
    g = torch.Generator("cuda").manual_seed(T)
    parts = torch.randn(S, T, N, generator=g, device="cuda")
    res = torch.randn(T, N, generator=g, device="cuda").to(torch.bfloat16) if resid else None
    w = torch.randn(N, generator=g, device="cuda").to(torch.bfloat16)
    out = ops.TiledAct(T, N, torch.device("cuda")) if tiled else None
    h, y = ops.reduce_residual_rmsnorm(parts, res, w, 1e-6, normed_out=out, want_hidden=hidden)
    y = y.to_rows() if tiled else y
    cut = [slice(a, min(a + 148, T)) for a in range(0, T, 148)]
    want = [ops.reduce_residual_rmsnorm(parts[:, c].contiguous(), None if res is None else res[c].contiguous(), w, 1e-6) for c in cut]
    if hidden:
        assert torch.equal(h, torch.cat([a for a, _ in want]))
    ref = torch.cat([b for _, b in want])
    # the sum of squares is taken in another order: the scale moves by a few 2^-24, a result by one bf16 step at most
    assert ((y.float() - ref.float()).abs() <= ref.float().abs() * 2.0 ** -7).all()


@pytest.mark.parametrize("page,hq,hkv,D", [(128, 24, 8, 128), (16, 16, 8, 64), (64, 12, 4, 128), (128, 16, 1, 64), (16, 32, 2, 128), (16, 16, 1, 128), (48, 18, 6, 64)])
def test_paged_attention_runs_of_rows(ops, page, hq, hkv, D):
    """Cache rows copied by twos, fours and singly: lengths around the ends of runs, slabs and tiles, against 64 bits; what lies behind a row's end in its page is never seen."""
    g = torch.Generator("cuda").manual_seed(page + hq)
    lens = [*range(1, 20), 31, 32, 33, 47, 48, 49, 63, 64, 65, 127, 128, 129, 400]
    pages = [(n + page - 1) // page for n in lens]
    kv = torch.randn(sum(pages), 2, page, hkv, D, generator=g, device="cuda").to(torch.bfloat16)
    q = torch.randn(len(lens), hq, D, generator=g, device="cuda").to(torch.bfloat16)
    order = torch.randperm(sum(pages), generator=g, device="cuda").tolist()
    indptr = [sum(pages[:i]) for i in range(len(lens) + 1)]
    want = []
    for i, n in enumerate(lens):
        own = order[indptr[i]:indptr[i + 1]]
        kv[own[-1], :, (n - 1) % page + 1:] = 100.0
        k, v = (kv[own, j].reshape(-1, hkv, D)[:n].double().repeat_interleave(hq // hkv, 1) for j in range(2))
        w = torch.softmax(torch.einsum("hd,khd->hk", q[i].double(), k) * D ** -0.5, -1)
        want.append(torch.einsum("hk,khd->hd", w, v))
    want = torch.stack(want)
    chunk = ops.attn_chunk_tokens(page, hkv)
    plan = ops.plan_rows(ops.RowPlan(len(lens), "cuda"), None, _i32(indptr), _i32(order), _i32([(n - 1) % page + 1 for n in lens]), len(lens), len(lens), page, chunk)
    ws = ops.paged_attn_workspace(len(lens), None, hq, hkv, D, "cuda")
    for grid in (None, 1, 7):
        out = ops.paged_attn(q, kv, 0, plan, len(lens), hkv, page, chunk, ws, grid_ctas=grid)
        _close(out, want, 2.0 ** -8)               # weights rounded to bf16, then the result: 2^-9 each at most


@pytest.mark.parametrize("page,hkv,D", [(16, 2, 64), (16, 2, 128), (16, 4, 64), (32, 1, 128)])
def test_paged_attention_bits_whatever_the_runs(ops, page, hkv, D):
    """A head's result does not depend on how the cache rows were copied: with twelve heads to a key head they come singly, with four by fours."""
    g, B = torch.Generator("cuda").manual_seed(page + D), 600
    lens = torch.randint(1, 40 * page, (B,), generator=g, device="cuda").tolist()
    pages = [(n + page - 1) // page for n in lens]
    kv = torch.randn(sum(pages), 2, page, hkv, D, generator=g, device="cuda").to(torch.bfloat16)
    q = torch.randn(B, hkv, 12, D, generator=g, device="cuda").to(torch.bfloat16)
    indptr = [sum(pages[:i]) for i in range(B + 1)]
    chunk = ops.attn_chunk_tokens(page, hkv)
    plan = ops.plan_rows(ops.RowPlan(B, "cuda"), None, _i32(indptr), _i32(list(range(sum(pages)))), _i32([(n - 1) % page + 1 for n in lens]), B, B, page, chunk)

    def run(q):
        hq = q.shape[1] * q.shape[2]
        ws = ops.paged_attn_workspace(B, None, hq, hkv, D, "cuda")
        return ops.paged_attn(q.reshape(B, hq, D).contiguous(), kv, 0, plan, B, hkv, page, chunk, ws, grid_ctas=100).view(B, hkv, -1, D)

    whole = run(q)
    for first in (0, 4, 8):
        assert torch.equal(run(q[:, :, first:first + 4]), whole[:, :, first:first + 4])


@pytest.mark.parametrize("hq,hkv,D", [(32, 2, 64), (16, 2, 128), (16, 1, 64), (24, 8, 128)])
def test_paged_attention_many_short_rows(ops, hq, hkv, D):
    """Rows of a tile or less behind one another in a CTA: every row with its own Q, however often (the next row's came too early now and then)."""
    g, page, B = torch.Generator("cuda").manual_seed(hq + hkv), 128, 96
    lens = [1 + 7 * i % 128 for i in range(B)]
    kv = torch.randn(B, 2, page, hkv, D, generator=g, device="cuda").to(torch.bfloat16)
    q = torch.randn(B, hq, D, generator=g, device="cuda").to(torch.bfloat16)
    k, v = (kv[:, j].double().repeat_interleave(hq // hkv, 2) for j in range(2))
    s = torch.einsum("bhd,bkhd->bhk", q.double(), k) * D ** -0.5
    s = s.masked_fill(torch.arange(page, device="cuda") >= torch.tensor(lens, device="cuda")[:, None, None], -float("inf"))
    want = torch.einsum("bhk,bkhd->bhd", torch.softmax(s, -1), v)
    chunk = ops.attn_chunk_tokens(page, hkv)
    plan = ops.plan_rows(ops.RowPlan(B, "cuda"), None, _i32(list(range(B + 1))), _i32(list(range(B))), _i32(lens), B, B, page, chunk)
    ws = ops.paged_attn_workspace(B, None, hq, hkv, D, "cuda")
    for grid in (1, 3, 7, 20):
        for _ in range(20):
            out = ops.paged_attn(q, kv, 0, plan, B, hkv, page, chunk, ws, grid_ctas=grid)
            err = (out.double() - want).flatten(1).norm(dim=1) / want.flatten(1).norm(dim=1)
            assert err.max() < 2.0 ** -8, (grid, lens[int(err.argmax())])      # weights rounded to bf16, then the result: 2^-9 each at most


@pytest.mark.parametrize("T,N,S,resid,tiled", [(1, 8, 2, True, False), (3, 264, 9, False, True), (64, 1032, 8, True, True), (65, 1024, 3, True, True), (148, 2048, 16, True, False),
                                               (130, 4096, 7, True, True), (149, 8, 1, True, False), (300, 1032, 3, False, True), (258, 2056, 2, True, True), (259, 3080, 1, False, False),
                                               (300, 4096, 5, True, True), (67, 4104, 2, True, False)])
def test_reduce_residual_rmsnorm_rows(ops, T, N, S, resid, tiled):
    """A thread to 8 columns up to 148 rows, beyond 128 threads to a row with one to four groups of columns; past 4096 columns the clusters."""
    g = torch.Generator("cuda").manual_seed(T)
    parts = torch.randn(S, T, N, generator=g, device="cuda")
    res = torch.randn(T, N, generator=g, device="cuda").to(torch.bfloat16) if resid else None
    w = torch.randn(N, generator=g, device="cuda").to(torch.bfloat16)
    out = ops.TiledAct(T, N, torch.device("cuda")) if tiled else None
    h, y = ops.reduce_residual_rmsnorm(parts, res, w, 1e-6, normed_out=out)
    y = y.to_rows() if tiled else y
    acc = parts[0].clone()
    for p in parts[1:]:
        acc += p
    want = acc.to(torch.bfloat16) if res is None else res + acc.to(torch.bfloat16)
    assert torch.equal(h, want)                                      # (the planes are added in their order)
    # against 64 bits: a sum of N squares in fp32 is off by less than 2^-13 of itself (its chains are shorter than 2^10 terms), the scale by half of that; then bf16
    hd = h.double()
    ref = hd * torch.rsqrt((hd * hd).mean(1, keepdim=True) + 1e-6) * w.double()
    assert ((y.double() - ref).abs() <= ref.abs() * (2.0 ** -8 + 2.0 ** -13)).all()


def _squares(h, parts):
    """Sums of the rows' squares in 32 bits, in order: with ``parts`` blocks to a row a thread takes 4 columns of every 1024 of its part, with 0 a lane 8 of every 256."""
    T, N = h.shape
    tree = lambda v: v[..., 0] if v.shape[-1] == 1 else tree(v[..., :v.shape[-1] // 2] + v[..., v.shape[-1] // 2:])          # noqa: E731
    pad = lambda v, n: torch.nn.functional.pad(v, (0, -v.shape[-1] % n))                                                     # noqa: E731
    if parts == 0:
        v = pad(h, 256).view(T, -1, 32, 4, 2)
        v = v[..., 0] * v[..., 0] + v[..., 1] * v[..., 1]              # (squares of bf16 values are exact)
        ss = torch.zeros(T, 32, device=h.device)
        for g in range(v.shape[1]):
            for j in range(4):
                ss = ss + v[:, g, :, j]
        return tree(ss)
    v = pad(h.view(T, parts, N // parts), 1024).view(T, parts, -1, 256, 4)
    ss = torch.zeros(T, parts, 256, device=h.device)
    for g in range(v.shape[2]):
        for j in range(4):
            ss = ss + v[:, :, g, :, j] * v[:, :, g, :, j]
    ss, total = tree(tree(ss.view(T, parts, 8, 32))), torch.zeros(T, device=h.device)
    for p in range(parts):
        total = total + ss[:, p]
    return total


@pytest.mark.parametrize("T", [1, 33, 64, 65, 128, 129, 148, 149, 192, 193, 512, 513, 1000])
@pytest.mark.parametrize("N", [8, 264, 1032, 2048, 3072, 4096])
def test_reduce_residual_rmsnorm_order_of_squares(ops, T, N):
    """The bits of the norm: a row's squares are added in one order for a number of rows, which rows off the 16-byte boundaries (another kernel) have as well."""
    g = torch.Generator("cuda").manual_seed(T + N)
    parts, w = torch.randn(3, T, N, generator=g, device="cuda"), torch.randn(N, generator=g, device="cuda").to(torch.bfloat16)
    res = torch.randn(T * N + 8, generator=g, device="cuda").to(torch.bfloat16)
    shifted = res.roll(4)[4:4 + T * N].view(T, N)                      # (8 bytes off)
    res = res[:T * N].view(T, N)
    assert torch.equal(res, shifted) and shifted.data_ptr() % 16 == 8
    h, y = ops.reduce_residual_rmsnorm(parts, res, w, 1e-6)
    split = next(c for c in (8, 4, 2, 1) if c <= (8 if T <= 64 else 4 if T <= 128 else 2 if T <= 192 else 1) and N % (4 * c) == 0)
    total = _squares(h.float(), 0 if T > 512 else split)
    rcp = torch.rsqrt(total / torch.full_like(total, N) + 1e-6)[:, None]
    assert torch.equal(y, (h.float() * rcp * w.float()).to(torch.bfloat16))
    if T <= 512:
        for a, b in zip((h, y), ops.reduce_residual_rmsnorm(parts, shifted, w, 1e-6)):
            assert torch.equal(a, b)


@pytest.mark.parametrize("T,dim,tiled", [(1, 8, False), (3, 2056, False), (65, 3072, True), (130, 8192, True), (2, 8200, False)])
def test_embedding_rmsnorm(ops, T, dim, tiled):
    """The same bits as the two launches; ids off the table's ends are taken to them; rows past 8192 columns take the two."""
    g = torch.Generator("cuda").manual_seed(dim)
    table, w = (torch.randn(n, dim, generator=g, device="cuda").to(torch.bfloat16) for n in (50, 1))
    ids = torch.randint(-3, 53, (T,), generator=g, device="cuda", dtype=torch.int32)
    hidden, normed = torch.empty(T, dim, device="cuda", dtype=torch.bfloat16), ops.TiledAct(T, dim, "cuda") if tiled else torch.empty(T, dim, device="cuda", dtype=torch.bfloat16)
    ops.embedding_rmsnorm(table, ids, w[0], 1e-6, hidden, normed)
    assert torch.equal(hidden, table[ids.clamp(0, 49).long()])
    assert torch.equal(normed.to_rows() if tiled else normed, ops.rmsnorm(hidden, w[0], 1e-6))


def _rotated(parts, bias, pos, freq, n_rot, D):
    """q | k | v rows of planes [S, T, (n_rot + n_v) D]: summed in order, biased and rounded, and with their first n_rot heads turned in 64 bits; and how far fp32 may be
    off them: angles, cosines and sines a few 2^-23 of one, the products and their sum as much of the larger, the result half a step of bf16 (8 bits: 2^-8 of itself at most)."""
    x = parts[0].clone()
    for p in parts[1:]:
        x += p
    x = (x if bias is None else x + bias.float()).to(torch.bfloat16).double().view(x.shape[0], -1, 2, D // 2)
    turn = (pos.float()[:, None] * freq).double().view(-1, 1, 2, D // 2)          # (the angle in 32 bits, as its rounding is large for late positions)
    c, s = turn.cos(), turn.sin()
    y = torch.stack((x[:, :, 0] * c[:, :, 0] - x[:, :, 1] * s[:, :, 0], x[:, :, 1] * c[:, :, 1] + x[:, :, 0] * s[:, :, 1]), 2)
    off = y.abs() * 2.0 ** -8 + x.abs().sum(2, keepdim=True) * 2.0 ** -20
    y[:, n_rot:], off[:, n_rot:] = x[:, n_rot:], 0.0
    return y.flatten(2), off.flatten(2)


@pytest.mark.parametrize("T,n_q,n_kv,D,S,bias", [(1, 1, 1, 16, 1, False), (3, 24, 8, 128, 3, True), (33, 5, 1, 80, 4, False), (64, 14, 2, 64, 5, True), (256, 2, 2, 256, 8, False),
                                                 (17, 3, 2, 16, 2, True), (129, 2, 1, 80, 3, True), (65, 1, 2, 256, 4, True)])
def test_qkv_rope_append_few_rows(ops, T, n_q, n_kv, D, S, bias):
    """Up to 256 rows (a row's items over blocks, four planes at a time) against 64 bits, and against the same rows in a step of 300: the same bits; a row without a page is not
    stored."""
    g = torch.Generator("cuda").manual_seed(T)
    page, W, R = 16, (n_q + 2 * n_kv) * D, 300
    parts = torch.randn(S, R, W, generator=g, device="cuda")
    freq = torch.rand(D, generator=g, device="cuda")
    b = torch.randn(W, generator=g, device="cuda").to(torch.bfloat16) if bias else None
    pos = torch.randint(0, 4000, (R,), generator=g, device="cuda", dtype=torch.int32)
    row_page, row_slot = torch.arange(R, device="cuda", dtype=torch.int32) // page, torch.arange(R, device="cuda", dtype=torch.int32) % page
    row_page[T // 2] = -1

    def run(n):
        kv, q = torch.zeros((R + page - 1) // page, 2, page, n_kv, D, device="cuda", dtype=torch.bfloat16), torch.zeros(R, n_q, D, device="cuda", dtype=torch.bfloat16)
        p = parts[:, :n].contiguous()
        ops.call("vb_qkv_rope_append", q.data_ptr(), kv.data_ptr(), p.data_ptr(), S, pos.data_ptr(), freq.data_ptr(), row_page.data_ptr(), row_slot.data_ptr(), n, n_q, n_kv, D,
                 page, D, 0, None, None, 0.0, None if b is None else b.data_ptr(), ops._stream())
        return q[:T], kv.transpose(1, 2).reshape(-1, 2, n_kv, D)[:T]

    got = run(T)
    for a, want in zip(got, run(R)):
        assert torch.equal(a, want)
    want, off = _rotated(parts[:, :T], b, pos[:T], freq, n_q + n_kv, D)
    kv = got[1].double()
    assert not kv[T // 2].any()
    stored = torch.arange(T, device="cuda") != T // 2
    have = torch.cat((got[0].double(), kv[:, 0], kv[:, 1]), 1)
    assert ((have - want).abs() <= off)[stored].all() and ((have - want).abs() <= off)[:, :n_q].all()


@pytest.mark.parametrize("T,n_q,n_kv,D,S,bias", [(257, 1, 1, 16, 1, False), (300, 24, 8, 128, 1, False), (258, 5, 1, 80, 3, True), (600, 2, 2, 256, 2, False)])
def test_qkv_rope_append_many_rows(ops, T, n_q, n_kv, D, S, bias):
    """A step of more than 256 rows against 64 bits, and against the same rows in steps of at most 200, which take the kernel of few rows; rows without a page keep the cache as
    it is."""
    g = torch.Generator("cuda").manual_seed(T)
    W, page = (n_q + 2 * n_kv) * D, 16
    parts = torch.randn(S, T, W, generator=g, device="cuda")
    b = torch.randn(W, generator=g, device="cuda").to(torch.bfloat16) if bias else None
    freq = (1.0 / 10000 ** (torch.arange(D, device="cuda") % (D // 2) / (D // 2))).float()
    pos = torch.randint(0, 4096, (T,), generator=g, device="cuda", dtype=torch.int32)
    n_pages = (T + page - 1) // page
    plan = ops.RowPlan(T, "cuda")
    at = torch.randperm(n_pages * page, generator=g, device="cuda")[:T].int()
    plan.row_page[:T] = at // page
    plan.row_slot[:T] = at % page
    plan.row_page[T // 2] = -1
    kv = [torch.full((n_pages, 2, page, n_kv, D), 7.0, dtype=torch.bfloat16, device="cuda") for _ in range(2)]
    q = ops.qkv_rope_append(parts, kv[0], pos, freq, plan, n_q, n_kv, D, qkv_bias=b)
    want = []
    for a in range(0, T, 200):
        n = min(200, T - a)
        sub = ops.RowPlan(n, "cuda")
        sub.row_page[:n] = plan.row_page[a:a + n]
        sub.row_slot[:n] = plan.row_slot[a:a + n]
        want.append(ops.qkv_rope_append(parts[:, a:a + n].contiguous(), kv[1], pos[a:a + n].contiguous(), freq, sub, n_q, n_kv, D, qkv_bias=b))
    # the same products and one sum, which the compiler may fuse on either side: one bf16 step of the larger term at most
    for got, ref in ((q, torch.cat(want)), (kv[0], kv[1])):
        assert ((got.float() - ref.float()).abs() <= ref.float().abs() * 2.0 ** -7 + 2.0 ** -20 * 8).all()
    want, off = _rotated(parts, b, pos, freq, n_q + n_kv, D)
    rows = kv[0].transpose(1, 2).reshape(-1, 2, n_kv, D).double()
    assert (rows == 7.0).flatten(1).all(1).sum() == n_pages * page - (T - 1)
    stored = torch.arange(T, device="cuda") != T // 2
    have = torch.cat((q.double(), rows[at.long(), 0], rows[at.long(), 1]), 1)
    assert ((have - want).abs() <= off)[stored].all() and ((have - want).abs() <= off)[:, :n_q].all()


@pytest.mark.parametrize("penalty", [1.3, 0.7, 3.0, 1.0 + 2.0 ** -23, 2.0 - 2.0 ** -23, 1e-3, 2.0 ** 39, 2.0 ** 41])
def test_sampler_quotients(ops, penalty):
    """The sampler's quotient of every positive bf16 against the division of the stand-alone penalty kernel: a penalised token ties
    with a token that already holds the divided value (the smaller index wins a tie) whichever of the two comes first."""
    code = torch.arange(1, 0x7f80, device="cuda").to(torch.int16).view(torch.bfloat16)
    n = code.numel()
    seen = torch.ones(n, 1, 1, 1, dtype=torch.bool, device="cuda")
    div = ops.apply_repetition_penalty(code.view(n, 1, 1), seen, penalty).view(n)
    for first in (0, 1):
        pair = torch.stack([code, div] if first == 0 else [div, code], 1).contiguous()
        mark = torch.zeros(n, 1, 1, 2, dtype=torch.bool, device="cuda")
        mark[..., first] = True
        assert (ops.sample(pair, "greedy", rep_cache=mark, penalty=penalty) == 0).all()

# logits a and b whose quotients by t are the same bf16 value; reciprocal and corrections give another one for a, since the remainders of such
# dividends lie below the smallest fp32 value
@pytest.mark.parametrize("a,b,t", [(2.7506567809241528e-36, 2.7624117244323756e-36, 1.0830623507415704e-12), (5.571843222897643e-36, 5.5953531099140885e-36, 1.3514122546715024e-12),
                                   (4.490388420141138e-36, 4.513898307157584e-36, 1.893335098077098e-12)])
def test_sampler_quotients_of_tiny_values(ops, a, b, t):
    x = torch.tensor([[a, b, a, b]], device="cuda").bfloat16().repeat(64, 1)          # (four: a token of a unit past the vocabulary takes the division)
    q = (x.cpu().float() / torch.full_like(x.cpu().float(), t)).bfloat16()      # (divided: a scalar divisor may be taken as a factor)
    assert (q == q[0, 0]).all()
    ids = ops.sample(x, "top_k", top_k=1, temperature=t, seed=3)                 # a tie: all are drawn
    assert set(ids.flatten().tolist()) == {0, 1, 2, 3}


@pytest.mark.parametrize("V", [1, 3, 4, 6, 2047, 4098, 40964, 81925, 156940])
@pytest.mark.parametrize("strategy", ["greedy", "top_p", "top_k_top_p", "min_p"])
def test_sampler_row_layouts(ops, V, strategy):
    """Rows on every boundary -- read four tokens, two, or one at a time -- give the same tokens; values that the quotient cannot take from the
    reciprocal, infinities and NaNs among them; the first unit, a remainder of every size, a last thread without a token."""
    g = torch.Generator("cuda").manual_seed(V)
    R = 5
    x = (torch.randn(R, V, generator=g, device="cuda") * 3).bfloat16()
    if V > 6:
        x[0, 1], x[1, 2], x[2, 3], x[3, :5], x[4, V - 1] = 0.0, -float("inf"), float("nan"), 2.0 ** -130, 3.0e38
        x[4, V - 2] = -3.0e38
    cache = torch.rand(R, 2, 1, V, generator=g, device="cuda") < 0.1
    kw = dict(top_p=0.8, top_k=7, min_p=0.05, temperature=0.6, penalty=1.3, seed=11, rep_cache=cache)
    want = ops.sample(x, strategy, **kw)
    for pad in (1, 2, 3, 4, 7):
        wide = torch.full((R, V + pad), float("nan"), device="cuda").bfloat16()
        wide[:, :V] = x
        assert torch.equal(ops.sample(wide[:, :V], strategy, **kw), want), pad
    if strategy == "greedy":
        y = ops.apply_repetition_penalty(x.view(R, 1, V), cache, 1.3).view(R, V).float().nan_to_num(nan=-float("inf"), posinf=float("inf"), neginf=-float("inf"))
        assert torch.equal(want.view(-1), y.argmax(-1))


@pytest.mark.parametrize("rows,dim,tiled", [(1, 8, False), (3, 2040, False), (33, 2056, True), (1, 3072, True), (2, 8192, False), (2, 8200, False)])
def test_rmsnorm_rows(ops, rows, dim, tiled):
    """Rows on 16-byte boundaries against the same rows with weights that are not, which take the general kernel."""
    g = torch.Generator("cuda").manual_seed(dim)
    x = torch.randn(rows, dim, generator=g, device="cuda").to(torch.bfloat16)
    w = torch.randn(dim + 1, generator=g, device="cuda").to(torch.bfloat16)
    out = ops.TiledAct(rows, dim, torch.device("cuda")) if tiled else None
    got = ops.rmsnorm(x, w[1:].clone(), 1e-5, out=out)
    assert torch.equal(got.to_rows() if tiled else got, ops.rmsnorm(x, w[1:], 1e-5))


def test_a_wait_that_runs_out_is_reported(ops):
    """The limit counts from the moment the block's gate opens; the flag reaches the host and the next call."""
    from vox_serve_b200 import _lib

    for pause in (0, 20000):                             # a wait of twenty times the limit in front of the gate is not late
        _lib.call("vb_wait_check", 1000, pause, 1, ops._stream())
    torch.cuda.synchronize()
    ops.check_waits()
    _lib.call("vb_wait_check", 1000, 0, 0, ops._stream())
    torch.cuda.synchronize()
    with pytest.raises(_lib.VoxB200Error, match="vb_wait_check"):
        ops.check_waits()
    ops.check_waits()
    _lib.call("vb_wait_check", 1000, 0, 0, ops._stream())
    torch.cuda.synchronize()
    with pytest.raises(_lib.VoxB200Error, match="ran out"):
        _lib.call("vb_wait_check", 1000, 0, 1, ops._stream())
    with pytest.raises(_lib.VoxB200Error, match="outside"):
        _lib.call("vb_wait_check", -1, 0, 1, ops._stream())


def test_warps_agree_on_a_wait_that_ran_out(ops):
    """One warp's wait runs out, the other's does not: both meet, and both know."""
    import ctypes

    from vox_serve_b200 import _lib

    flags = (ctypes.c_ubyte * 8).from_address(_lib.load().vb_wait_flags())
    at = _lib.WAIT_KINDS.index("vb_wait_check")
    for complete in (1, 0, 1):
        _lib.call("vb_wait_check", 1000, 100, complete, ops._stream())
        torch.cuda.synchronize()
        assert flags[at] == (0 if complete else 3)
        flags[at] = 0


def test_snac_decoder_that_ends_wide(monkeypatch):
    """A decoder whose last convolution has more channels than the channels-last one takes decodes channel-first."""
    from vox_serve_b200.tokenizer.snac import SNAC

    out = []
    for plain in ("0", "1"):
        monkeypatch.setenv("VB_SNAC_FP32", plain)
        m = SNAC(decoder_dim=1024, decoder_rates=(4,), device="cuda")
        m.load_state_dict(m.synthetic_state_dict(5))
        codes = [torch.arange(n, device="cuda")[None] for n in (2, 4, 8)]
        out.append(m.decode(codes, noises=[torch.zeros(*s, device="cuda") for s in m.noise_shapes(1, 8)]))
    _close(out[0], out[1].double(), 1e-4)                # (tf32 halves cut off at 2^-20 beside plain 32-bit products)
