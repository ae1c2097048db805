"""Each CUDA kernel alone against a plain float32 (or float64) torch restatement of the
same operation, at sizes other than the tiny models': widths that are no power of two,
head sizes in steps of 16, odd head counts and groups, scattered pages, windows."""
import ctypes
import math

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda:0"


def ops():
    from tgo_b200.kernels import ops as o
    return o


def attention_part():
    """The module that picks the attention kernel for a step."""
    from tgo_b200.parts import attention
    return attention


def rnd(*shape, dtype=torch.float32, scale=1.0, seed=0):
    g = torch.Generator(device="cpu").manual_seed(seed)
    return (torch.randn(*shape, generator=g) * scale).to(dtype).to(DEV)


def tol(dtype):
    return dict(rtol=2e-2, atol=2e-2) if dtype == torch.bfloat16 else dict(rtol=2e-5, atol=2e-5)


# --------------------------------------------------------------------- elementwise


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_embed(dtype):
    table = rnd(1000, 200, dtype=dtype)
    ids = torch.tensor([0, 999, 17, 17, 501], dtype=torch.int32, device=DEV)
    out = torch.empty(5, 200, dtype=torch.float32, device=DEV)
    ops().embed(table, ids, out)
    assert torch.equal(out, table[ids.long()].float())


@pytest.mark.parametrize("d", [72, 200, 4096, 5120, 20000])
@pytest.mark.parametrize("act", [torch.float32, torch.bfloat16])
def test_add_rmsnorm(d, act):
    T, eps = 5, 1e-5
    h = rnd(T, d, seed=1)
    delta = rnd(T, d, dtype=act, seed=2)
    gain = 1 + 0.1 * rnd(d, seed=3)
    want_h = h + delta.float()
    want = (want_h * torch.rsqrt((want_h * want_h).mean(-1, keepdim=True) + eps)) * gain
    out = torch.empty(T, d, dtype=act, device=DEV)
    h2 = h.clone()
    ops().add_rmsnorm(h2, delta, gain, eps, out)
    assert torch.allclose(h2, want_h, rtol=0, atol=1e-6)
    assert torch.allclose(out.float(), want, **tol(act))
    # no delta
    out2 = torch.empty(T, d, dtype=act, device=DEV)
    h3 = h.clone()
    ops().add_rmsnorm(h3, None, gain, eps, out2)
    want2 = (h * torch.rsqrt((h * h).mean(-1, keepdim=True) + eps)) * gain
    assert torch.equal(h3, h) and torch.allclose(out2.float(), want2, **tol(act))
    # selected rows: h stays, the add happens on the fly
    rows = torch.tensor([4, 0, 4], dtype=torch.int32, device=DEV)
    out3 = torch.empty(3, d, dtype=act, device=DEV)
    h4 = h.clone()
    ops().add_rmsnorm(h4, delta, gain, eps, out3, rows)
    assert torch.equal(h4, h) and torch.allclose(out3.float(), want[rows.long()], **tol(act))


@pytest.mark.parametrize("f,T", [(88, 7), (200, 1), (12288, 3), (1001, 2)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_swiglu(f, T, dtype):
    gu = rnd(T, 2 * f, dtype=dtype, scale=2.0)
    out = torch.empty(T, f, dtype=dtype, device=DEV)
    ops().swiglu(gu, out)
    g, u = gu[:, :f].float(), gu[:, f:].float()
    want = g / (1 + torch.exp(-g)) * u
    assert torch.allclose(out.float(), want, **tol(dtype))
    if f % 8 == 0:
        v = gu.reshape(T, f // 8, 2, 8)
        g, u = v[:, :, 0].reshape(T, f).float(), v[:, :, 1].reshape(T, f).float()
        ops().swiglu(gu, out, interleaved=True)
        assert torch.allclose(out.float(), g / (1 + torch.exp(-g)) * u, **tol(dtype))


def rope_ref(x, pos, theta, rot):
    half = rot // 2
    inv = theta ** (-2.0 * torch.arange(half, dtype=torch.float64, device=x.device) / rot)
    ang = pos.double()[:, None] * inv[None, :]
    cos, sin = ang.cos().float()[:, None, :], ang.sin().float()[:, None, :]
    y = x.clone()
    lo, hi = x[..., :half], x[..., half:rot]
    y[..., :half] = lo * cos - hi * sin
    y[..., half:rot] = lo * sin + hi * cos
    return y


@pytest.mark.parametrize("H,Hkv", [(8, 2), (5, 1), (32, 8), (3, 3)])
def test_qk_norm_rope_cache_many_tokens(H, Hkv):
    """Head size 128, bfloat16, a prompt portion's worth of tokens: the kernel with half a
    warp per head vector (head counts that leave half-warps idle or mix q, k and v in a warp)."""
    T, ps, pages, eps, theta, dh = 70, 16, 9, 1e-6, 1e6, 128
    dtype = torch.bfloat16
    qkv = rnd(T, (H + 2 * Hkv) * dh, dtype=dtype, seed=H)
    q, k, v = qkv[:, :H * dh], qkv[:, H * dh:(H + Hkv) * dh], qkv[:, (H + Hkv) * dh:]
    qg, kg = 1 + 0.1 * rnd(dh, seed=5), 1 + 0.1 * rnd(dh, seed=6)
    pos = torch.arange(300, 300 + T, dtype=torch.int32, device=DEV)
    slot_list = [(5 * t + 3) % (pages * ps) if t != 11 else -1 for t in range(T)]     # scattered, one padded
    assert len({s for s in slot_list if s >= 0}) == T - 1
    slots = torch.tensor(slot_list, dtype=torch.int32, device=DEV)
    inv = (theta ** (-2.0 * torch.arange(dh // 2, dtype=torch.float64) / dh)).to(DEV)
    kc = torch.zeros(pages, Hkv, ps, dh, dtype=dtype, device=DEV)
    vc = torch.zeros_like(kc)

    def norm(x, g):
        x = x.float()
        return (x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps)) * g
    want_q = rope_ref(norm(q.reshape(T, H, dh), qg), pos, theta, dh)
    want_k = rope_ref(norm(k.reshape(T, Hkv, dh), kg), pos, theta, dh)
    want_v = v.reshape(T, Hkv, dh).clone()
    table = ops().rope_table(pos, inv)
    ops().qk_norm_rope_cache(q, k, v, H, Hkv, dh, qg, kg, eps, table, dh, slots, kc, vc, ps)
    assert torch.allclose(q.reshape(T, H, dh).float(), want_q, **tol(dtype))
    for t in range(T):
        s = slot_list[t]
        if s < 0:
            continue
        assert torch.allclose(kc[s // ps, :, s % ps].float(), want_k[t], **tol(dtype))
        assert torch.equal(vc[s // ps, :, s % ps], want_v[t])
    written = {s for s in slot_list if s >= 0}
    for s in range(pages * ps):
        if s not in written:
            assert not kc[s // ps, :, s % ps].any() and not vc[s // ps, :, s % ps].any()


@pytest.mark.parametrize("H,Hkv,dh,rot", [(5, 5, 16, 16), (6, 2, 48, 32), (8, 1, 128, 128),
                                          (3, 3, 80, 80)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_qk_norm_rope_cache(H, Hkv, dh, rot, dtype):
    T, ps, pages, eps, theta = 9, 4, 12, 1e-5, 5e5
    width = (H + 2 * Hkv) * dh
    qkv = rnd(T, width, dtype=dtype)
    q, k, v = qkv[:, :H * dh], qkv[:, H * dh:(H + Hkv) * dh], qkv[:, (H + Hkv) * dh:]
    qg, kg = 1 + 0.1 * rnd(dh, seed=5), 1 + 0.1 * rnd(dh, seed=6)
    pos = torch.tensor([0, 1, 2, 3, 100, 101, 7, 4000, 9], dtype=torch.int32, device=DEV)
    slots = torch.tensor([4, 5, 6, 7, 40, 41, -1, 13, 47], dtype=torch.int32, device=DEV)
    inv = (theta ** (-2.0 * torch.arange(rot // 2, dtype=torch.float64) / rot)).to(DEV)
    kc = torch.zeros(pages, Hkv, ps, dh, dtype=dtype, device=DEV)
    vc = torch.zeros_like(kc)

    def norm(x, g):
        x = x.float()
        return (x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps)) * g
    want_q = rope_ref(norm(q.reshape(T, H, dh), qg), pos, theta, rot)
    want_k = rope_ref(norm(k.reshape(T, Hkv, dh), kg), pos, theta, rot)
    want_v = v.reshape(T, Hkv, dh).clone()
    table = ops().rope_table(pos, inv)
    ops().qk_norm_rope_cache(q, k, v, H, Hkv, dh, qg, kg, eps, table, rot, slots, kc, vc, ps)
    assert torch.allclose(q.reshape(T, H, dh).float(), want_q, **tol(dtype))
    for t in range(T):
        s = int(slots[t])
        if s < 0:
            continue
        assert torch.allclose(kc[s // ps, :, s % ps].float(), want_k[t], **tol(dtype))
        assert torch.equal(vc[s // ps, :, s % ps], want_v[t])
    written = {int(s) for s in slots if s >= 0}
    for s in range(pages * ps):
        if s not in written:
            assert not kc[s // ps, :, s % ps].any() and not vc[s // ps, :, s % ps].any()


@pytest.mark.parametrize("M,N,K", [(1, 5, 7), (3, 130, 96), (70, 65, 33), (129, 257, 1000)])
def test_sgemm(M, N, K):
    x, w = rnd(M, K, seed=1), rnd(N, K, seed=2)
    out = torch.empty(M, N, device=DEV)
    ops().sgemm_tn(x, w, out)
    want = (x.double() @ w.double().t()).float()
    assert torch.allclose(out, want, rtol=1e-5, atol=1e-4)
    # a row's result does not depend on the rows beside it
    out1 = torch.empty(1, N, device=DEV)
    ops().sgemm_tn(x[M - 1:M].contiguous(), w, out1)
    assert torch.equal(out1[0], out[M - 1])


@pytest.mark.parametrize("M,N,K", [(1, 1, 1), (15, 63, 17), (17, 65, 16), (64, 128, 50), (65, 129, 64), (200, 68, 33)])
def test_sgemm_tiles(M, N, K):
    """Every tile gives a sum over k in order: the same bits."""
    from tgo_b200.kernels.build import load_library
    x, w = rnd(M, K, seed=3), rnd(N, K, seed=4)
    outs = []
    try:
        for tile in (1, 2, 3):
            load_library("sgemm").tgo_sgemm_force_tile(tile)
            outs.append(torch.full((M, N), float("nan"), device=DEV))
            ops().sgemm_tn(x, w, outs[-1])
    finally:
        load_library("sgemm").tgo_sgemm_force_tile(0)
    want = x.double() @ w.double().t()
    # a chain of K roundings of at most K |x| |w| 2^-24 each
    bound = K * 2.0 ** -24 * (x.double().abs() @ w.double().abs().t())
    assert ((outs[0].double() - want).abs() <= bound + 1e-30).all()
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])


@pytest.mark.parametrize("M,N,K", [(1, 1, 256), (31, 127, 260), (33, 129, 576), (64, 128, 640), (97, 257, 1020), (161, 130, 2048),
                                   (330, 40, 6144)])
def test_sgemm_by_parts(M, N, K):
    """Three bfloat16 parts a number: the same bits from every tile and beside any rows, an error below that of a
    chain of FMA, and the plain kernel's result where one is not finite."""
    from tgo_b200.kernels.build import load_library
    lib = load_library("sgemm")
    x, w = rnd(M, K, seed=5), rnd(N, K, seed=6)
    assert lib.tgo_sgemm_part_bytes(ctypes.c_void_p(w.data_ptr()), K, N) > 0
    outs = []
    try:
        for columns in (160, 128, 96, 64, 32, 0):
            lib.tgo_sgemm_force_columns(columns)
            outs.append(torch.full((M, N), float("nan"), device=DEV))
            ops().sgemm_tn(x, w, outs[-1])
    finally:
        lib.tgo_sgemm_force_columns(0)
    assert all(torch.equal(o, outs[0]) for o in outs)
    last = torch.empty(1, N, device=DEV)
    ops().sgemm_tn(x[M - 1:].contiguous(), w, last)
    assert torch.equal(last[0], outs[0][M - 1])
    # a k-block of 64: four cuts of less than 2^-23 of its sum's size, the products left out (2^-26 a term)
    # and a rounded addition: K / 64 times 2^-21 of the sum of sizes is above all of them
    want, size = x.double() @ w.double().t(), x.double().abs() @ w.double().abs().t()
    assert ((outs[0].double() - want).abs() <= (K + 63) // 64 * 2.0 ** -21 * size).all()
    plain, got = torch.empty(M, N, device=DEV), torch.empty(M, N, device=DEV)
    if M * N > 1000:
        # that bound is one of the worst case, which two parts a number (2-norm 4e-6) stay below as well: three err by 1.3e-7
        # (K = 2048) to 1.9e-7 (6144), and by no more than a chain of FMA
        try:
            lib.tgo_sgemm_force_tile(1)
            ops().sgemm_tn(x, w, plain)
        finally:
            lib.tgo_sgemm_force_tile(0)
        err = (outs[0].double() - want).norm()
        assert err <= 4e-7 * want.norm() and err <= (plain.double() - want).norm()
    x[M // 2, 3], x[M - 1, K - 1], w[N // 2, 7] = float("inf"), float("nan"), -3.4e38
    x[0, 7] = 1e-3
    ops().sgemm_tn(x, w, got)
    try:
        lib.tgo_sgemm_force_tile(1)
        ops().sgemm_tn(x, w, plain)
    finally:
        lib.tgo_sgemm_force_tile(0)
    odd = ~torch.isfinite(plain)
    assert torch.equal(torch.isfinite(got), ~odd)
    assert torch.equal(got[odd].nan_to_num(7.0), plain[odd].nan_to_num(7.0))
    assert torch.allclose(got[~odd], plain[~odd], rtol=1e-4, atol=1e-3)
    assert ops().sgemm_error() == 0


@pytest.mark.parametrize("up,wide", [(1e-38, 1.0), (1e-40, 1e3), (1e-36, 1e30), (1.0, 1e-39), (1e-22, 1e-22), (1e33, 1e-30),
                                     (1e25, 1e10)])
def test_sgemm_by_parts_small_and_large_numbers(up, wide):
    """Numbers whose lower parts have no bfloat16 number of their size, and sizes past those the parts are scaled for."""
    M, N, K = 33, 130, 512
    x, w = (rnd(M, K, seed=5).double() * up).float(), (rnd(N, K, seed=6).double() * wide).float()
    y = torch.empty(M, N, device=DEV)
    ops().sgemm_tn(x, w, y)
    want, size = x.double() @ w.double().t(), x.double().abs() @ w.double().abs().t()
    # the bound of the parts, or a chain's of K roundings; a rounding below the normal numbers is 2^-150 at most
    assert ((y.double() - want).abs() <= K * 2.0 ** -24 * size + K * 2.0 ** -150).all()
    if up < 1e20:                                        # by parts: all three of them, and one rounding to a number that may be no normal one
        assert (y.double() - want).norm() <= 4e-7 * want.norm() + (M * N) ** 0.5 * 2.0 ** -149


def test_sgemm_by_parts_takes_a_bounded_workspace(monkeypatch):
    """Rows whose parts together are past the bound go in groups: the same bits, two launches each, within it."""
    o, M, N, K = ops(), 1001, 300, 1024
    x, w = rnd(M, K, seed=5), rnd(N, K, seed=6)
    want, got = torch.empty(M, N, device=DEV), torch.empty(M, N, device=DEV)
    o.sgemm_tn(x, w, want)
    for rows, goes in ((400, 3), (1, 1001), (1001, 1)):
        monkeypatch.setattr(o, "SGEMM_PARTS_BYTES", 6 * K * rows)
        torch.cuda.synchronize()
        torch.cuda.reset_peak_memory_stats()
        before, launches = torch.cuda.memory_allocated(), o.LAUNCHES[0]
        o.sgemm_tn(x, w, got.fill_(float("nan")))
        torch.cuda.synchronize()
        assert torch.cuda.max_memory_allocated() - before <= 6 * K * rows + 512 and o.LAUNCHES[0] - launches == 2 * goes
        assert torch.equal(got, want)
    monkeypatch.setattr(o, "SGEMM_PARTS_BYTES", 0)
    o.sgemm_tn(x[:3].contiguous(), w, got[:3])
    assert torch.equal(got[:3], want[:3])


@pytest.mark.parametrize("M,N,K", [(1, 1, 256), (40, 200, 1000), (557, 2048, 2048)])
def test_sgemm_by_parts_past_their_range(M, N, K):
    """Every output of numbers that the parts are not scaled for: the plain kernel's bits, at a time of its kind (an output
    made by a thread for itself took 250 to 400 times as long as by parts; by tiles it is six to nine times)."""
    from tgo_b200.kernels.build import load_library
    lib, o = load_library("sgemm"), ops()
    x, w = rnd(M, K, seed=5) * 1e33, rnd(N, K, seed=6) * 1e-5
    x[:, 3] = 3e33                                       # every row has one past 2^103
    outs = [torch.empty(M, N, device=DEV) for _ in range(2)]
    assert lib.tgo_sgemm_part_bytes(ctypes.c_void_p(w.data_ptr()), K, N) > 0
    o.sgemm_tn(x, w, outs[0])
    try:
        lib.tgo_sgemm_force_tile(1)
        o.sgemm_tn(x, w, outs[1])
    finally:
        lib.tgo_sgemm_force_tile(0)
    inside = (x.double() * 2.0 ** 24 @ (w.double() * 2.0 ** 24).t()).abs() < 2.0 ** 127
    assert bool(torch.isfinite(outs[1]).all()) and not bool(inside.all())
    assert torch.equal(*outs) and o.sgemm_error() == 0

    if M > 500:
        small = x * 1e-33
        assert best_time(lambda: o.sgemm_tn(x, w, outs[0])) <= 20 * best_time(lambda: o.sgemm_tn(small, w, outs[0]))


@pytest.mark.parametrize("T,H,G,dk,dv,rot", [(1, 1, 1, 16, 16, 16), (11, 3, 1, 48, 32, 16), (130, 2, 2, 64, 128, 0),
                                             (1203, 16, 4, 128, 128, 64)])
def test_projection_rows_eight_channels_at_a_time(T, H, G, dk, dv, rot):
    """The form of whole runs of channels against 64 bits (a bfloat16 rounding of float32 arithmetic), tokens that
    are not stored among them, single tokens and fours."""
    o, ps = ops(), 16
    w = H * dk + G * (dk + dv)
    x = rnd(T, w, seed=dk).to(torch.bfloat16)
    bias = rnd(w, seed=3)
    rope = rnd(T, rot, seed=4) if rot else None
    slots = torch.randperm(T + 40, generator=torch.Generator().manual_seed(1))[:T].to(torch.int32).to(DEV)
    slots[T // 2] = -1
    pages = (T + 40 + ps - 1) // ps
    kc, vc = (torch.zeros((pages, G, ps, n), dtype=torch.bfloat16, device=DEV) for n in (dk, dv))
    y, at = (x.double() + bias.double()), [H * dk, H * dk + G * dk]

    def turned(z):
        if rot:
            c, s = rope[:, None, :rot // 2].double(), rope[:, None, rot // 2:].double()
            lo, hi = z[..., :rot // 2], z[..., rot // 2:rot]
            z = torch.cat([lo * c - hi * s, hi * c + lo * s, z[..., rot:]], -1)
        return z
    wq, wk, wv = turned(y[:, :at[0]].reshape(T, H, dk)), turned(y[:, at[0]:at[1]].reshape(T, G, dk)), y[:, at[1]:].reshape(T, G, dv)
    o.qkv_bias_rope_cache(x[:, :at[0]], x[:, at[0]:at[1]], x[:, at[1]:], H, G, dk, dv, bias[:at[0]].contiguous(),
                          bias[at[0]:at[1]].contiguous(), bias[at[1]:].contiguous(), rope, rot, False, slots, kc, vc, ps)
    close = lambda a, b: bool(((a.double() - b).abs() <= 2.0 ** -8 * b.abs() + 1e-5).all())    # noqa: E731
    assert close(x[:, :at[0]].reshape(T, H, dk), wq)
    stored = slots >= 0
    s = slots[stored].long()
    assert close(kc[s // ps, :, s % ps], wk[stored]) and close(vc[s // ps, :, s % ps], wv[stored])
    rest = torch.ones(pages * ps, dtype=torch.bool, device=DEV)
    rest[s] = False
    r = rest.nonzero().flatten()
    assert not kc[r // ps, :, r % ps].any() and not vc[r // ps, :, r % ps].any()


# ----------------------------------------------------------------------- attention


def paged_case(extents, firsts, H, Hkv, dh, ps, dtype, seed=0, crafted=None):
    """A ragged batch over a scattered paged cache. Returns the kernel inputs and the
    per-request dense keys and values."""
    g = torch.Generator().manual_seed(seed)
    B = len(extents)
    ctx_lens = [f + e for f, e in zip(firsts, extents)]
    n_pages = sum((c + ps - 1) // ps for c in ctx_lens) + 3
    perm = (torch.randperm(n_pages - 1, generator=g) + 1).tolist()      # page 0 stays unused
    width = max((c + ps - 1) // ps for c in ctx_lens)
    bt = torch.zeros(B, width, dtype=torch.int32)
    kc = torch.full((n_pages, Hkv, ps, dh), float("nan"))
    vc = torch.full((n_pages, Hkv, ps, dh), float("nan"))
    dense = []
    for b in range(B):
        K = torch.randn(ctx_lens[b], Hkv, dh, generator=g)
        V = torch.randn(ctx_lens[b], Hkv, dh, generator=g)
        if crafted is not None:
            crafted(b, K, V)
        K, V = K.to(dtype).float(), V.to(dtype).float()
        dense.append((K, V))
        for i in range((ctx_lens[b] + ps - 1) // ps):
            page = perm.pop()
            bt[b, i] = page
            n = min(ps, ctx_lens[b] - i * ps)
            kc[page, :, :n] = K[i * ps:i * ps + n].transpose(0, 1)
            vc[page, :, :n] = V[i * ps:i * ps + n].transpose(0, 1)
    T = sum(extents)
    q = torch.randn(T, H * dh, generator=g)
    pos, seq = [], []
    for b in range(B):
        pos += list(range(firsts[b], ctx_lens[b]))
        seq += [b] * extents[b]
    return dict(q=q.to(dtype).to(DEV), kc=kc.to(dtype).to(DEV), vc=vc.to(dtype).to(DEV),
                bt=bt.to(DEV), pos=torch.tensor(pos, dtype=torch.int32, device=DEV),
                seq=torch.tensor(seq, dtype=torch.int32, device=DEV), dense=dense,
                extents=extents, firsts=firsts)


def attention_ref(case, H, Hkv, dh, scale, window):
    q = case["q"].float().cpu()
    out = torch.zeros_like(q)
    t = 0
    G = H // Hkv
    for b, (e, f) in enumerate(zip(case["extents"], case["firsts"])):
        K, V = case["dense"][b]
        for i in range(e):
            p = f + i
            lo = max(0, p - window + 1) if window else 0
            for h in range(H):
                s = (K[lo:p + 1, h // G] @ q[t, h * dh:(h + 1) * dh]) * scale
                w = torch.softmax(s.double(), 0).float()
                out[t, h * dh:(h + 1) * dh] = w @ V[lo:p + 1, h // G]
            t += 1
    return out


class Ctx:
    """The fields of a StepContext that the attention dispatch reads."""

    def __init__(self, case, decode):
        self.extents = case["extents"]
        self.positions, self.seq_ids = case["pos"], case["seq"]
        self.token_ids = case["pos"]
        self.num_seqs = len(self.extents)
        self.max_context = max(f + e for f, e in zip(case["firsts"], case["extents"]))
        self.decode_only = decode
        self.aux = {}


class Cache:
    def __init__(self, case, ps):
        self.k, self.v, self.block_tables, self.page_size = case["kc"], case["vc"], case["bt"], ps


SHAPES = [(4, 2, 16, 16), (6, 2, 32, 8), (8, 8, 64, 16), (32, 8, 128, 16), (5, 1, 48, 4),
          (3, 3, 128, 32), (16, 2, 128, 16), (16, 1, 128, 8), (12, 2, 128, 64)]


@pytest.mark.parametrize("H,Hkv,dh,ps", SHAPES)
@pytest.mark.parametrize("window", [0, 37])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_attention_mixed_batch(H, Hkv, dh, ps, window, dtype):
    """Prompt portions beside single tokens, through whichever kernel the dispatch picks."""
    extents, firsts = [70, 1, 5, 1, 130], [0, 199, 61, 0, 100]
    case = paged_case(extents, firsts, H, Hkv, dh, ps, dtype, seed=H + dh)
    scale = 1 / math.sqrt(dh)
    want = attention_ref(case, H, Hkv, dh, scale, window)
    out = torch.zeros_like(case["q"])
    attention_part().paged_attention(case["q"], out, H, Hkv, dh, Cache(case, ps), Ctx(case, False), scale,
                          window)
    assert torch.allclose(out.float().cpu(), want, **tol(dtype))
    out2 = torch.zeros_like(case["q"])
    ops().attention_generic(case["q"], out2, H, Hkv, dh, case["kc"], case["vc"], ps, case["bt"],
                            case["seq"], case["pos"], scale, window)
    assert torch.allclose(out2.float().cpu(), want, **tol(dtype))


@pytest.mark.parametrize("H,Hkv,dh,ps", [(4, 4, 8, 4), (6, 2, 36, 8), (16, 1, 256, 16), (5, 1, 132, 32), (16, 4, 128, 16)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_attention_generic_tiles(H, Hkv, dh, ps, dtype, monkeypatch):
    """Keys through shared memory for a block of queries: the bits of a warp a query, with every
    option, requests that meet inside a block, and a token that brings nothing."""
    case = paged_case([33, 1, 7, 64], [0, 40, 31, 5], H, Hkv, dh, ps, dtype, seed=dh)
    case["pos"][-1] = -1
    T = case["q"].shape[0]
    extra = dict(sinks=rnd(H, seed=1), softcap=3.0, dist_bias=rnd(50, H, seed=2), gate=rnd(T, H, seed=3).to(dtype))
    for kw in ({}, extra):
        outs = []
        for start in (4, 10 ** 9):
            monkeypatch.setattr(ops(), "GENERIC_TILES_FROM", start)
            outs.append(torch.full_like(case["q"], 7.0))
            ops().attention_generic(case["q"], outs[-1], H, Hkv, dh, case["kc"], case["vc"], ps, case["bt"],
                                    case["seq"], case["pos"], dh ** -0.5, 0, **kw)
        assert torch.equal(outs[0], outs[1]) and bool(torch.isfinite(outs[0].float()).all())
        assert not outs[0][-1].any()


@pytest.mark.parametrize("H,Hkv", [(4, 4), (4, 2), (6, 2), (5, 1), (12, 2)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_attention_generic_tiles_keep_requests_apart(H, Hkv, dtype, monkeypatch):
    """Groups of heads that do not fill a warp's rows, requests that meet inside a warp, one of them with
    values that are not finite: the others' rows are finite and every row is that of a warp a query."""
    def crafted(b, K, V):
        if b == 1:
            V[0], V[1, :, ::2], V[5] = float("nan"), float("inf"), float("-inf")
    case = paged_case([6, 3, 1, 9, 2], [40, 35, 70, 0, 33], H, Hkv, 36, 8, dtype, seed=H, crafted=crafted)
    outs = []
    for start in (4, 10 ** 9):
        monkeypatch.setattr(ops(), "GENERIC_TILES_FROM", start)
        outs.append(torch.full_like(case["q"], 7.0))
        ops().attention_generic(case["q"], outs[-1], H, Hkv, 36, case["kc"], case["vc"], 8, case["bt"], case["seq"],
                                case["pos"], 36 ** -0.5, 0)
    others = case["seq"] != 1
    assert bool(torch.isfinite(outs[1][others].float()).all()) and bool(torch.isnan(outs[1][~others].float()).any())
    assert torch.equal(torch.isnan(outs[0]), torch.isnan(outs[1]))
    assert torch.equal(outs[0].nan_to_num(nan=5.0), outs[1].nan_to_num(nan=5.0))


@pytest.mark.parametrize("H,Hkv", [(4, 4), (6, 2), (16, 1)])
def test_attention_generic_tiles_in_any_order(H, Hkv, monkeypatch):
    """Tokens in no order, so that there are more runs of one request than requests: the same rows."""
    case = paged_case([33, 1, 7, 64], [0, 40, 31, 5], H, Hkv, 36, 8, torch.float32, seed=H)
    case["pos"][-1] = case["pos"][40] = -1
    order = torch.randperm(case["q"].shape[0], generator=torch.Generator().manual_seed(1)).to(DEV)
    outs = []
    for start, idx in ((10 ** 9, slice(None)), (4, order)):
        monkeypatch.setattr(ops(), "GENERIC_TILES_FROM", start)
        outs.append(torch.full_like(case["q"], 7.0))
        ops().attention_generic(case["q"][idx].contiguous(), outs[-1], H, Hkv, 36, case["kc"], case["vc"], 8, case["bt"],
                                case["seq"][idx].contiguous(), case["pos"][idx].contiguous(), 36 ** -0.5, 0)
    assert torch.equal(outs[0][order], outs[1])


@pytest.mark.parametrize("H,Hkv,dh", [(8, 8, 64), (16, 4, 128)])
def test_attention_generic_tiles_beside_single_tokens(H, Hkv, dh, monkeypatch):
    """A prompt portion beside single tokens of long contexts: requests that meet in a block do not wait
    for each other's keys (when they did, 8/8 heads of 64 took 2691 us where a warp a query took 557)."""
    case = paged_case([64] + [1] * 15, [0] + [1000] * 15, H, Hkv, dh, 16, torch.float32)
    out, took = torch.empty_like(case["q"]), {}
    for start in (4, 10 ** 9):
        monkeypatch.setattr(ops(), "GENERIC_TILES_FROM", start)
        times = []
        for _ in range(5):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            for _ in range(4):
                ops().attention_generic(case["q"], out, H, Hkv, dh, case["kc"], case["vc"], 16, case["bt"], case["seq"],
                                        case["pos"], dh ** -0.5, 0)
            b.record()
            torch.cuda.synchronize()
            times.append(a.elapsed_time(b))
        took[start] = min(times)
    assert took[4] < took[10 ** 9], took


@pytest.mark.parametrize("H,Hkv,dh,ps", SHAPES)
@pytest.mark.parametrize("window", [0, 100])
def test_attention_decode_split(H, Hkv, dh, ps, window):
    """Decode-only batch in bfloat16: keys cut over several CTAs and joined."""
    extents, firsts = [1, 1, 1, 1], [0, 63, 64, 700]
    case = paged_case(extents, firsts, H, Hkv, dh, ps, torch.bfloat16, seed=3)
    scale = 1 / math.sqrt(dh)
    want = attention_ref(case, H, Hkv, dh, scale, window)
    for n_splits in (1, 2, 5, 8, 16):
        out = torch.zeros_like(case["q"])
        if not ops().flash_supports(dh, H // Hkv):
            pytest.skip("no tensor-core instance for this head size")
        ops().attention_flash(case["q"], out, H, Hkv, dh, case["kc"], case["vc"], ps, case["bt"],
                              case["pos"], case["seq"], None, None, scale, window,
                              n_splits=n_splits)
        assert torch.allclose(out.float().cpu(), want, **tol(torch.bfloat16)), n_splits


@pytest.mark.parametrize("H,Hkv,ps", [(32, 8, 16), (3, 3, 32), (16, 2, 8), (16, 1, 64), (12, 2, 16)])
@pytest.mark.parametrize("window", [0, 100])
@pytest.mark.parametrize("norm,rotate", [(True, True), (False, True), (True, False)])
def test_attention_decode_fused_equals_the_two_kernels(H, Hkv, ps, window, norm, rotate):
    """The decode kernel that norms, rotates and stores the step's own q, k and v itself gives
    the bits of qk_norm_rope_cache followed by the decode kernel: in the attention's result
    and in the cache. The requests' own positions lie at the start, the end and the middle of
    a tile of 64 keys and of a page, and in every split."""
    dh = 128
    o = ops()
    extents, firsts = [1, 1, 1, 1, 1, 1], [0, 63, 64, 700, 255, 130]
    case = paged_case(extents, firsts, H, Hkv, dh, ps, torch.bfloat16, seed=H + ps)
    T = len(extents)
    g = torch.Generator().manual_seed(5)
    qkv = (torch.randn(T, (H + 2 * Hkv) * dh, generator=g) * 2).to(torch.bfloat16).to(DEV)
    qw, kw = H * dh, Hkv * dh
    q_gain = (1 + 0.3 * torch.randn(dh, generator=g)).to(DEV) if norm else None
    k_gain = (1 + 0.3 * torch.randn(dh, generator=g)).to(DEV) if norm else None
    rope = None
    if rotate:
        inv = torch.tensor([10000.0 ** (-2 * i / dh) for i in range(dh // 2)], dtype=torch.float64, device=DEV)
        rope = o.rope_table(case["pos"], inv)
    slots = torch.empty(T, dtype=torch.int32)
    for t in range(T):
        pos = firsts[t]
        slots[t] = int(case["bt"][t, pos // ps]) * ps + pos % ps
    slots = slots.to(DEV)
    scale = 1 / math.sqrt(dh)
    # the two kernels
    a = qkv.clone()
    kc1, vc1 = case["kc"].clone(), case["vc"].clone()
    o.qk_norm_rope_cache(a[:, :qw], a[:, qw:qw + kw], a[:, qw + kw:], H, Hkv, dh, q_gain, k_gain, 1e-6,
                         rope, dh if rotate else 0, slots, kc1, vc1, ps)
    for n_splits in (1, 3, 8):
        want = torch.zeros(T, qw, dtype=torch.bfloat16, device=DEV)
        o.attention_flash(a[:, :qw], want, H, Hkv, dh, kc1, vc1, ps, case["bt"], case["pos"], case["seq"],
                          None, None, scale, window, n_splits=n_splits)
        b = qkv.clone()
        kc2, vc2 = case["kc"].clone(), case["vc"].clone()
        assert o.decode_attention_fuses(b[:, :qw], dh, H // Hkv, ps, kc2, vc2, dh if rotate else 0)
        got = torch.zeros(T, qw, dtype=torch.bfloat16, device=DEV)
        o.attention_decode_fused(b[:, :qw], b[:, qw:qw + kw], b[:, qw + kw:], got, H, Hkv, dh, q_gain,
                                 k_gain, 1e-6, rope, slots, kc2, vc2, ps, case["bt"], case["pos"],
                                 case["seq"], scale, window, n_splits=n_splits)
        bits = lambda t: t.view(torch.int16)               # unwritten rows of the cache hold NaN
        assert torch.equal(bits(kc2), bits(kc1)) and torch.equal(bits(vc2), bits(vc1)), n_splits
        assert torch.equal(bits(got), bits(want)), n_splits
        assert torch.equal(b, qkv)                         # the raw rows are left as they came
    assert o.attention_decode_tma_error() == 0


@pytest.mark.parametrize("far", [0, 15, 16, 63, 64, 127, 128, 499])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("dh", [64, 128])
def test_attention_far_key_stands_out(far, dtype, dh):
    """One key among 500 is made to carry nearly all the weight; a kernel that skips it (a
    tile's or a page's edge) returns something else entirely. Head size 64 goes through the
    mma.sync kernels, 128 (in bfloat16) through the tcgen05 kernel for the portion and the
    TMA-fed kernel for the single token."""
    H, Hkv, ps = 8, 2, 16

    def crafted(b, K, V):
        K *= 0.05
        K[far] = 0
        K[far, :, 0] = 30.0
        V[far] = 7.0
    case = paged_case([1, 12], [499, 488], H, Hkv, dh, ps, dtype, seed=far, crafted=crafted)
    q = torch.zeros_like(case["q"])
    q[:, 0::dh] = 8.0                       # channel 0 of every head
    case["q"] = q
    scale = 1 / math.sqrt(dh)
    out = torch.zeros_like(q)
    attention_part().paged_attention(q, out, H, Hkv, dh, Cache(case, ps), Ctx(case, False), scale, 0)
    sees = case["pos"] >= far                # rows before the far key cannot read it
    assert sees.any()
    assert torch.allclose(out[sees].float(), torch.full_like(out[sees], 7.0).float(), atol=0.05)
    out = torch.zeros_like(q[:1])
    case1 = dict(case, q=q[:1], pos=case["pos"][:1], seq=case["seq"][:1], extents=[1], firsts=[499])
    attention_part().paged_attention(q[:1], out, H, Hkv, dh, Cache(case, ps), Ctx(case1, True), scale, 0)
    assert torch.allclose(out.float(), torch.full_like(out, 7.0).float(), atol=0.05)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("H,Hkv,dh,ps", [(4, 2, 32, 8), (8, 2, 128, 16), (32, 8, 128, 16)])
def test_attention_window_edge(dtype, H, Hkv, dh, ps):
    """The key just outside the window carries a huge score and must not be read; the key
    just inside must be. (Head size 128 in bfloat16: the TMA-fed decode kernel, and the
    tcgen05 kernel when the token comes as a portion.)"""
    W = 40
    p = 200
    for edge, expect in ((p - W, 1.0), (p - W + 1, 7.0)):
        def crafted(b, K, V, edge=edge):
            K *= 0.01
            V[:] = 1.0
            K[edge, :, 0] = 50.0
            V[edge] = 7.0
        case = paged_case([1], [p], H, Hkv, dh, ps, dtype, seed=1, crafted=crafted)
        q = torch.zeros_like(case["q"])
        q[:, 0::dh] = 8.0
        for decode in (True, False):
            out = torch.zeros_like(q)
            attention_part().paged_attention(q, out, H, Hkv, dh, Cache(case, ps), Ctx(case, decode),
                                  1 / math.sqrt(dh), W)
            assert torch.allclose(out.float(), torch.full_like(out, expect).float(), atol=0.05)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("H,Hkv,dh,ps", [(4, 2, 32, 8), (8, 2, 128, 16), (32, 8, 128, 16), (6, 2, 64, 32)])
def test_attention_window_edge_inside_a_portion(dtype, H, Hkv, dh, ps):
    """A prompt portion of 121 tokens at positions 140..260 with a window of 40, so the
    window's start moves through the kernel's key tiles row by row. Key 170 carries a huge
    score and the value 7, every other value is 1: exactly the rows at positions 170..209
    may read it (earlier rows are before it, later rows' windows have passed it)."""
    W, first, n, edge = 40, 140, 121, 170

    def crafted(b, K, V):
        K *= 0.01
        V[:] = 1.0
        K[edge, :, 0] = 50.0
        V[edge] = 7.0
    case = paged_case([n], [first], H, Hkv, dh, ps, dtype, seed=4, crafted=crafted)
    q = torch.zeros_like(case["q"])
    q[:, 0::dh] = 8.0
    out = torch.zeros_like(q)
    attention_part().paged_attention(q, out, H, Hkv, dh, Cache(case, ps), Ctx(case, False),
                                     1 / math.sqrt(dh), W)
    pos = torch.arange(first, first + n, device=DEV)
    sees = (pos >= edge) & (pos - W + 1 <= edge)
    want = torch.where(sees, 7.0, 1.0)[:, None].expand_as(out)
    bad = (out.float() - want).abs().amax(dim=1) > 0.05
    assert not bad.any(), f"wrong at positions {pos[bad].tolist()}"


def test_attention_unusual_head_size_falls_back():
    """Head sizes without a tensor-core instance run through the generic kernel."""
    H, Hkv, dh, ps = 4, 2, 80, 16
    case = paged_case([33, 1], [0, 50], H, Hkv, dh, ps, torch.bfloat16)
    want = attention_ref(case, H, Hkv, dh, 0.1, 0)
    out = torch.zeros_like(case["q"])
    attention_part().paged_attention(case["q"], out, H, Hkv, dh, Cache(case, ps), Ctx(case, False), 0.1, 0)
    assert torch.allclose(out.float().cpu(), want, **tol(torch.bfloat16))


def test_kernels_refuse_what_they_cannot_take():
    o = ops()
    q = torch.zeros(1, 4 * 528, dtype=torch.float32, device=DEV)
    with pytest.raises(o.KernelError):
        o.qk_norm_rope_cache(q, None, None, 4, 4, 528, None, None, 1e-6, None, 0, None, None,
                             None, 0)
    with pytest.raises(o.KernelError):
        o.embed(torch.zeros(4, 4), torch.zeros(1, dtype=torch.int32), torch.zeros(1, 4))


# ------------------------------------------------------------------------ sampling


def test_argmax_lowest_id_on_ties():
    logits = torch.zeros(3, 151936, device=DEV)
    logits[0, 77] = 5.0
    logits[0, 150000] = 5.0
    logits[1, 151935] = 1.0
    out = torch.empty(3, dtype=torch.int32, device=DEV)
    ops().argmax(logits, out)
    assert out.tolist() == [77, 151935, 0]


@pytest.mark.parametrize("V", [1000, 151936])
@pytest.mark.parametrize("policy", [dict(temperature=0.8), dict(temperature=1.3, top_k=40),
                                    dict(temperature=0.7, top_p=0.9),
                                    dict(temperature=1.0, top_k=128, top_p=0.5),
                                    dict(temperature=0.0)])
def test_sample_matches_plain(V, policy):
    import plain_qwen3 as plain
    n = 6
    logits = rnd(n, V, scale=3.0, seed=V)
    draws = [0.0, 0.13, 0.5, 0.77, 0.999, 0.31]
    out = torch.empty(n, dtype=torch.int32, device=DEV)
    ops().sample(logits, torch.full((n,), policy.get("temperature", 0.0), device=DEV),
                 torch.full((n,), policy.get("top_k", 0), dtype=torch.int32, device=DEV),
                 torch.full((n,), policy.get("top_p", 0.0), device=DEV),
                 torch.tensor(draws, device=DEV), out)
    host = logits.cpu().numpy()
    for r in range(n):
        ids, w, total = plain.policy_distribution(host[r], **policy)
        want = plain.walk(ids, w, total, draws[r])
        got = int(out[r])
        if got == want:
            continue
        # The device sums the weights in another order than the plain single ascending
        # float32 sum; over 150k terms the two running sums differ by about 1e-4 of the
        # total, which moves a boundary by a few ids. The chosen id must be a kept one whose
        # interval of the exact (float64) distribution lies within that distance of the draw.
        assert got in ids, f"row {r}: {got} is not a kept id"
        cdf = np.cumsum(np.asarray(w, np.float64))
        target = draws[r] * cdf[-1]
        i = ids.index(got)
        lo = cdf[i - 1] if i > 0 else 0.0
        slack = 5e-4 * cdf[-1]
        assert lo - slack <= target <= cdf[i] + slack, (r, got, want)


@pytest.mark.parametrize("V", [300, 151936])
@pytest.mark.parametrize("policy", [dict(temperature=0.8), dict(temperature=1.3, top_k=40),
                                    dict(temperature=0.7, top_p=0.9),
                                    dict(temperature=1.0, top_k=3, top_p=0.99),
                                    dict(temperature=0.0)])
def test_sample_reports_the_distribution_it_drew_from(V, policy):
    """The report of sample: the drawn token's share of the kept weights and the most likely
    alternatives, against the plain distribution in float64; rows that ask for nothing stay
    untouched, and asking changes no draw."""
    import plain_qwen3 as plain
    n = 6
    logits = rnd(n, V, scale=3.0, seed=V + 1)
    logits[2, 17] = logits[2, 5] = logits[2].max() + 1          # a tie at the top: lower id first
    draws = [0.0, 0.13, 0.5, 0.77, 0.999, 0.31]
    wants = [0, 5, 128, -1, 1, 20]
    args = (logits, torch.full((n,), policy.get("temperature", 0.0), device=DEV),
            torch.full((n,), policy.get("top_k", 0), dtype=torch.int32, device=DEV),
            torch.full((n,), policy.get("top_p", 0.0), device=DEV), torch.tensor(draws, device=DEV))
    quiet = torch.empty(n, dtype=torch.int32, device=DEV)
    ops().sample(*args, quiet)
    out = torch.empty(n, dtype=torch.int32, device=DEV)
    lp = torch.full((n,), 7.0, device=DEV)
    top_ids = torch.full((n, 128), -1, dtype=torch.int32, device=DEV)
    top_lp = torch.full((n, 128), 7.0, device=DEV)
    ops().sample(*args, out, torch.tensor(wants, dtype=torch.int32, device=DEV), lp, top_ids, top_lp)
    assert out.tolist() == quiet.tolist()
    host = logits.cpu().numpy()
    for r, w_ in enumerate(wants):
        if w_ < 0:
            assert float(lp[r]) == 7.0 and int(top_ids[r, 0]) == -1
            continue
        # the oracle's totals are float64 sums: the plain single ascending float32 sum is
        # itself 1e-4 off over 150k terms, the device's (per thread, then over the threads in
        # order) about 1e-6
        ids, w, total = plain.policy_distribution(host[r], exact_totals=True, **policy)
        got = int(out[r])
        want_lp, want_top = plain.token_logprobs(ids, w, total, got, w_, V)
        assert got in ids and np.isfinite(float(lp[r]))          # a drawn token is a kept one
        assert abs(float(lp[r]) - want_lp) < 2e-5, (r, float(lp[r]), want_lp)
        k = min(w_, V)
        got_ids, got_lp = top_ids[r, :k].tolist(), top_lp[r, :k].tolist()
        assert int(top_ids[r, k]) == -1 if k < 128 else True
        assert all(a >= b for a, b in zip(got_lp, got_lp[1:])), r
        for j, ((i, v), gi, gv) in enumerate(zip(want_top, got_ids, got_lp)):
            if v == -np.inf:
                assert gv == -np.inf and gi == i, (r, j)
            else:
                assert abs(gv - v) < 2e-5, (r, j, gv, v)
                # equal ids, but for neighbours whose float32 weights are within rounding
                assert gi == i or abs(host[r][gi] - host[r][i]) < 1e-5 * abs(host[r][i]), (r, j)
        if r == 2 and w_ >= 2 and policy.get("temperature", 0.0) > 0:
            assert got_ids[:2] == [5, 17]
        if policy.get("top_k", 0) and k >= policy["top_k"]:
            kept = min(policy["top_k"], len(ids))
            assert abs(sum(math.exp(v) for v in got_lp[:kept]) - 1) < 1e-4
            assert all(v == -np.inf for v in got_lp[kept:])


def test_logits_adjust_matches_plain():
    import plain_qwen3 as plain
    V = 500
    row = rnd(V, scale=2.0, seed=9)
    history = [3, 3, 7, 499, 3, 0]
    want = plain.penalize(row.cpu().numpy() + 0, history, rep=1.3, presence=0.5, frequency=0.25)
    want[11] += 0  # no bias on 11
    from tgo_b200.sampling.policy import Policy
    from tgo_b200.sampling.sampler import adjust_row
    pol = Policy(repetition_penalty=1.3, presence_penalty=0.5, frequency_penalty=0.25,
                 logit_bias={5: -2.0})
    base = row.cpu().numpy().copy()
    base[5] += -2.0
    want = plain.penalize(base, history, rep=1.3, presence=0.5, frequency=0.25)
    adjust_row(row, pol, history)
    assert np.allclose(row.cpu().numpy(), want, rtol=1e-6, atol=1e-6)


# ------------------------------------------------------------- weight-streaming GEMM


# at most 8 rows, 256 or more rows of W and a K that is a multiple of 2048 go to the persistent
# form (one CTA an SM, x staged in shared memory) unless x is too large for that (8 x 12288);
# the rest to the form of one CTA a 16-row tile
@pytest.mark.parametrize("M,N,K", [(1, 16, 64), (3, 50, 96), (8, 257, 224), (9, 64, 4096),
                                   (16, 100, 1000), (17, 33, 72), (40, 48, 512), (64, 130, 264),
                                   (1, 256, 2048), (5, 4099, 2048), (8, 6144, 520), (7, 300, 72),
                                   (8, 2500, 4096), (2, 1000, 12288), (8, 304, 12288),
                                   (3, 777, 6144)])
def test_gemm_skinny(M, N, K):
    x = rnd(M, K, dtype=torch.bfloat16, seed=1)
    w = rnd(N, K, dtype=torch.bfloat16, scale=0.1, seed=2)
    want = x.float() @ w.float().t()
    for dt in (torch.bfloat16, torch.float32):
        out = torch.empty(M, N, dtype=dt, device=DEV)
        ops().gemm_skinny(x, w, out)
        assert torch.allclose(out.float(), want, rtol=1e-2 if dt == torch.bfloat16 else 1e-4,
                              atol=2e-2 if dt == torch.bfloat16 else 1e-3), (M, N, K, dt)
    h = rnd(M, N, seed=3)
    h2 = h.clone()
    ops().gemm_skinny(x, w, h2, accumulate=True)
    assert torch.allclose(h2, h + want, rtol=1e-4, atol=1e-3)
    # a row's result does not depend on the rows beside it (bit for bit while the same form of
    # the kernel takes both: the two forms cut K differently)
    out_all = torch.empty(M, N, dtype=torch.float32, device=DEV)
    ops().gemm_skinny(x, w, out_all)
    out_one = torch.empty(1, N, dtype=torch.float32, device=DEV)
    ops().gemm_skinny(x[M - 1:M].contiguous(), w, out_one)
    if ops().folds_norm(M, N, K) == ops().folds_norm(1, N, K):
        assert torch.equal(out_one[0], out_all[M - 1])
    else:
        assert torch.allclose(out_one[0], out_all[M - 1], rtol=1e-4, atol=1e-3)


def interleave8(gate, up):
    f, d = gate.shape
    return torch.stack([gate.view(f // 8, 8, d), up.view(f // 8, 8, d)], dim=1).reshape(2 * f, d)


@pytest.mark.parametrize("M,f,K", [(2, 224, 64), (8, 128, 96), (16, 1000, 264), (8, 1000, 2048),
                                   (3, 688, 4096)])
def test_gemm_skinny_gated_output(M, f, K):
    """A gate/up matrix with rows interleaved in eights: the kernel applies the gate itself."""
    x = rnd(M, K, dtype=torch.bfloat16, seed=4)
    wg = rnd(f, K, dtype=torch.bfloat16, scale=0.2, seed=5)
    wu = rnd(f, K, dtype=torch.bfloat16, scale=0.2, seed=6)
    g = (x.float() @ wg.float().t()).to(torch.bfloat16).float()
    u = (x.float() @ wu.float().t()).to(torch.bfloat16).float()
    want = g / (1 + torch.exp(-g)) * u
    w = interleave8(wg, wu).contiguous()
    out = torch.empty(M, f, dtype=torch.bfloat16, device=DEV)
    ops().gemm_skinny(x, w, out, gated=True)
    assert torch.allclose(out.float(), want, rtol=2e-2, atol=2e-2)
    # the separate kernel on the interleaved product gives the same
    gu = (x.float() @ w.float().t()).to(torch.bfloat16)
    out2 = torch.empty(M, f, dtype=torch.bfloat16, device=DEV)
    ops().swiglu(gu, out2, interleaved=True)
    assert torch.allclose(out2.float(), want, rtol=2e-2, atol=2e-2)
    # and gated_linear picks either
    got = ops().gated_linear(x, w, True)
    assert torch.allclose(got.float(), want, rtol=2e-2, atol=2e-2)


@pytest.mark.parametrize("M,N,K", [(1, 256, 2048), (5, 4099, 2048), (8, 6144, 4096), (8, 1008, 4096),
                                   (3, 304, 8192), (2, 320, 6144)])
def test_gemm_skinny_with_the_norm_folded_in(M, N, K):
    """RMSNorm of the float32 stream made while the product stages its rows: against the
    norm kernel followed by the product, and against float64."""
    o = ops()
    assert o.folds_norm(M, N, K) and not o.folds_norm(8, 4096, 12288) and not o.folds_norm(2, 64, 2048)
    assert not o.folds_norm(8, 5120, 5120) and o.folds_norm(4, 4096, 12288)
    h = rnd(M, K, scale=3.0, seed=11)
    h[M - 1, 5] = 400.0                                        # a row with its own scale
    gain = 1 + rnd(K, scale=0.2, seed=12)
    w = rnd(N, K, dtype=torch.bfloat16, scale=0.1, seed=13)
    lazy = o.NormedRows(h, gain, 1e-5, torch.bfloat16)
    x = torch.empty(M, K, dtype=torch.bfloat16, device=DEV)
    o.add_rmsnorm(h, None, gain, 1e-5, x)
    hd = h.double()
    exact = (hd * torch.rsqrt((hd * hd).mean(1, keepdim=True) + 1e-5) * gain.double())
    want = exact.to(torch.bfloat16).double() @ w.double().t()
    for dt in (torch.bfloat16, torch.float32):
        sep = torch.empty(M, N, dtype=dt, device=DEV)
        o.gemm_skinny(x, w, sep)
        got = torch.empty(M, N, dtype=dt, device=DEV)
        o.gemm_skinny_normed(lazy, w, got)
        # the two norms add their squares in another order: a row of x may differ by one
        # bfloat16 step in a few places
        tol = 2e-2 if dt == torch.bfloat16 else 2e-3
        assert torch.allclose(got.double(), want, rtol=tol, atol=tol * want.abs().max().item())
        assert torch.allclose(got.float(), sep.float(), rtol=tol, atol=tol * want.abs().max().item())
        assert torch.equal(o.linear(lazy, w, dt), got)          # linear folds it the same way
    assert torch.equal(lazy.rows(), x)                          # and what does not fold asks for the rows
    # a row's result does not depend on the rows beside it
    one = torch.empty(1, N, dtype=torch.float32, device=DEV)
    o.gemm_skinny_normed(o.NormedRows(h[M - 1:].contiguous(), gain, 1e-5, torch.bfloat16), w, one)
    assert torch.equal(one[0], got[M - 1])
    if N % 16 == 0:
        gated = torch.empty(M, N // 2, dtype=torch.bfloat16, device=DEV)
        o.gemm_skinny_normed(lazy, w, gated, gated=True)
        sep = torch.empty(M, N // 2, dtype=torch.bfloat16, device=DEV)
        o.gemm_skinny(x, w, sep, gated=True)
        assert torch.allclose(gated.float(), sep.float(), rtol=3e-2, atol=3e-2 * sep.float().abs().max().item())
        assert torch.equal(o.gated_linear(lazy, w, True), gated)


# ------------------------------------------------------------------ tcgen05 product


def tc_flag():
    return int(ops().gemm_tc_error_flag(DEV).item())


@pytest.mark.parametrize("M,N,K", [
    (128, 128, 64), (200, 300, 264), (700, 520, 1000), (1024, 2048, 4096), (300, 512, 2048),
    (2048, 4096, 192), (2048, 6144, 128), (130, 1001, 72), (33, 200, 264), (8, 128, 64)])
def test_gemm_tc(M, N, K):
    """The tcgen05 kernel with tails in every dimension."""
    x = rnd(M, K, dtype=torch.bfloat16, seed=M + K)
    w = rnd(N, K, dtype=torch.bfloat16, scale=0.1, seed=N + K)
    want = x.float() @ w.float().t()
    atol = 3 * 2.0 ** -8.5 * math.sqrt(K) * 0.1 + 1e-3         # float32 accumulation of exact bf16 products
    for dt in (torch.float32, torch.bfloat16):
        out = torch.zeros(M, N, dtype=dt, device=DEV)
        ops().gemm_tc(x, w, out)
        torch.cuda.synchronize()
        assert tc_flag() == 0
        if dt == torch.float32:
            assert torch.allclose(out, want, rtol=1e-4, atol=1e-3), (M, N, K)
        else:
            assert torch.allclose(out.float(), want, rtol=1e-2, atol=atol + 2e-2)
    h = rnd(M, N, seed=3)
    h2 = h.clone()
    ops().gemm_tc(x, w, h2, accumulate=True)
    assert torch.allclose(h2, h + want, rtol=1e-4, atol=1e-3) and tc_flag() == 0


@pytest.mark.parametrize("M,f,K", [(300, 512, 264), (1000, 1000, 512), (24, 256, 512), (64, 1008, 264)])
def test_gemm_tc_gated_output(M, f, K):
    x = rnd(M, K, dtype=torch.bfloat16, seed=4)
    wg = rnd(f, K, dtype=torch.bfloat16, scale=0.2, seed=5)
    wu = rnd(f, K, dtype=torch.bfloat16, scale=0.2, seed=6)
    g = (x.float() @ wg.float().t()).to(torch.bfloat16).float()
    u = (x.float() @ wu.float().t()).to(torch.bfloat16).float()
    want = g / (1 + torch.exp(-g)) * u
    out = torch.zeros(M, f, dtype=torch.bfloat16, device=DEV)
    ops().gemm_tc(x, interleave8(wg, wu).contiguous(), out, gated=True)
    torch.cuda.synchronize()
    assert tc_flag() == 0
    assert torch.allclose(out.float(), want, rtol=2e-2, atol=2e-2 * float(want.abs().max()))


@pytest.mark.parametrize("rows,width", [(128, 64), (128, 144), (128, 224), (128, 256), (256, 64),
                                        (256, 96), (256, 176), (256, 240), (256, 256)])
@pytest.mark.parametrize("M", [600, 700])
def test_gemm_tc_tile_shapes(rows, width, M):
    """Every kind of tile the kernel takes, forced instead of chosen: one accumulator or two
    (128 or 256 rows), narrow, odd and full widths, with tails in rows and columns (600 rows
    leave the lower accumulator of the last tile wholly outside, 700 partly); plain, added
    and gated outputs."""
    N, K = 1008, 328
    x = rnd(M, K, dtype=torch.bfloat16, seed=M)
    w = rnd(N, K, dtype=torch.bfloat16, scale=0.1, seed=width)
    want = x.float() @ w.float().t()
    ops().gemm_tc_force_tile(rows, width)
    try:
        out = torch.zeros(M, N, dtype=torch.float32, device=DEV)
        ops().gemm_tc(x, w, out)
        h = rnd(M, N, seed=3)
        h2 = h.clone()
        ops().gemm_tc(x, w, h2, accumulate=True)
        gated = torch.zeros(M, N // 2, dtype=torch.bfloat16, device=DEV)
        ops().gemm_tc(x, interleave8(w[:N // 2], w[N // 2:]).contiguous(), gated, gated=True)
        torch.cuda.synchronize()
    finally:
        ops().gemm_tc_force_tile(0, 0)
    assert tc_flag() == 0
    assert torch.allclose(out, want, rtol=1e-4, atol=1e-3)
    assert torch.allclose(h2, h + want, rtol=1e-4, atol=1e-3)
    g = want[:, :N // 2].to(torch.bfloat16).float()
    u = want[:, N // 2:].to(torch.bfloat16).float()
    act = g / (1 + torch.exp(-g)) * u
    assert torch.allclose(gated.float(), act, rtol=2e-2, atol=2e-2 * float(act.abs().max()))


@pytest.mark.parametrize("M,N,K,rows,width,parts", [
    (300, 512, 2048, 128, 256, 4),      # 6 tiles, each cut four ways
    (300, 512, 2048, 256, 128, 4),      # 8 tiles of two accumulators, cut four ways
    (2100, 2600, 1024, 128, 256, 2),    # 187 tiles: a full round, then 39 tiles cut in two
    (2100, 2600, 1024, 256, 256, 1),    # 99 tiles, fewer than SMs: no cut (148 / 99 < 2)
    (2100, 2600, 1536, 256, 176, 1),    # 135 tiles: no cut
    (1100, 2608, 1024, 256, 176, 1),    # 75 tiles: no cut
    (700, 1008, 4096, 256, 240, 8),     # 15 tiles cut eight ways (a part has 8 k-blocks at least)
    (520, 4000, 1280, 128, 112, 2)])    # 180 tiles: one round, the 32 left cut in two
def test_gemm_tc_cut_last_round(M, N, K, rows, width, parts):
    """The tiles of the last round, cut along K over the idle CTAs and joined through the
    workspace: the same results as without the cut (up to the order of float32 sums), in
    every output form, and again on a second launch (the flags went back to zero)."""
    x = rnd(M, K, dtype=torch.bfloat16, seed=M)
    w = rnd(N - N % 16, K, dtype=torch.bfloat16, scale=0.1, seed=width)
    N = w.shape[0]
    want = x.float() @ w.float().t()
    h = rnd(M, N, seed=3)
    wgu = interleave8(w[:N // 2], w[N // 2:]).contiguous()
    got = {}
    for cut in (False, True, True):
        ops().gemm_tc_force_tile(rows, width, cut_last_round=cut)
        try:
            out = torch.zeros(M, N, dtype=torch.float32, device=DEV)
            ops().gemm_tc(x, w, out)
            h2 = h.clone()
            ops().gemm_tc(x, w, h2, accumulate=True)
            ob = torch.zeros(M, N, dtype=torch.bfloat16, device=DEV)
            ops().gemm_tc(x, w, ob)
            gated = torch.zeros(M, N // 2, dtype=torch.bfloat16, device=DEV)
            ops().gemm_tc(x, wgu, gated, gated=True)
            torch.cuda.synchronize()
        finally:
            ops().gemm_tc_force_tile(0, 0)
        assert tc_flag() == 0
        if torch.cuda.get_device_properties(0).multi_processor_count == 148:
            assert ops().gemm_tc_last_plan() == (rows, width, parts if cut else 1)
        assert torch.allclose(out, want, rtol=1e-4, atol=1e-3)
        assert torch.allclose(h2, h + want, rtol=1e-4, atol=1e-3)
        if cut in got:      # the second launch with the cut: bit for bit the first
            for a, b in zip(got[cut], (out, h2, ob, gated)):
                assert torch.equal(a, b)
        got[cut] = (out, h2, ob, gated)
    assert torch.allclose(got[True][0], got[False][0], rtol=1e-5, atol=1e-4)
    assert torch.allclose(got[True][2].float(), got[False][2].float(), rtol=1e-2, atol=2e-2)
    assert torch.allclose(got[True][3].float(), got[False][3].float(), rtol=2e-2,
                          atol=2e-2 * float(got[False][3].float().abs().max()))
    flags = ops()._tc_tail_buffers(DEV)[1]
    assert int(flags.abs().sum().item()) == 0


def test_linear_picks_by_rows_and_agrees():
    """1..8 rows: the weight-streaming kernel; from TC_MIN_ROWS rows: tcgen05; between them
    the library. The same product through each differs by bfloat16 rounding only."""
    w = rnd(384, 512, dtype=torch.bfloat16, scale=0.1, seed=6)
    x = rnd(ops().TC_MIN_ROWS + 70, 512, dtype=torch.bfloat16, seed=7)
    many = ops().linear(x, w)
    mid = ops().linear(x[:40].contiguous(), w)
    few = ops().linear(x[:5].contiguous(), w)
    assert torch.allclose(many[:40].float(), mid.float(), rtol=2e-2, atol=2e-2)
    assert torch.allclose(many[:5].float(), few.float(), rtol=2e-2, atol=2e-2)
    assert tc_flag() == 0


# --------------------------------------------------------------------- attention on tcgen05


TC_CASES = [
    # extents, firsts, H, Hkv, page size, window
    ([32], [0], 4, 1, 16, 0),                               # one query tile, one key tile
    ([200], [0], 8, 2, 16, 0),                              # ragged last tile, two key tiles
    ([70, 1, 5, 1, 130], [0, 199, 61, 0, 100], 32, 8, 16, 0),      # portions beside single tokens
    ([70, 1, 5, 1, 130], [0, 199, 61, 0, 100], 32, 8, 16, 37),     # with a window
    ([300, 17], [50, 400], 3, 3, 32, 0),                    # no grouping, odd head count
    ([300], [0], 16, 1, 64, 100),                           # 16 heads a group, window over tiles
    ([513], [0], 8, 4, 128, 0),                             # a page as large as a key tile
    ([40], [1000], 8, 2, 8, 0),                             # small pages, a long context behind
    ([300, 9], [20, 0], 5, 1, 16, 0),                       # five heads a group: 25 tokens a tile, 3 rows idle
    ([200], [0], 6, 2, 32, 50),                             # three heads a group
    ([130], [70], 40, 8, 16, 0),                            # the 14B shape's heads
    ([40], [17000], 4, 1, 16, 0),                           # more pages than the on-chip table slice holds
    ([40], [17000], 4, 1, 16, 300),                         # the same behind a window
]


@pytest.mark.parametrize("extents,firsts,H,Hkv,ps,window", TC_CASES)
def test_attention_tc_prefill(extents, firsts, H, Hkv, ps, window):
    """The tcgen05 attention kernel alone (head size 128; one CTA per SM drawing items) over a
    scattered paged cache whose unwritten rows hold NaN, against the plain float32
    attention."""
    o, dh = ops(), 128
    assert o.attention_tc_supports(dh, H // Hkv, ps)
    case = paged_case(extents, firsts, H, Hkv, dh, ps, torch.bfloat16, seed=len(extents) + ps)
    scale = 1 / math.sqrt(dh)
    want = attention_ref(case, H, Hkv, dh, scale, window)
    out = torch.full_like(case["q"], float("nan"))
    tok0, ntok = attention_part().step_tiles(Ctx(case, False), 128 // (H // Hkv))
    o.attention_tc_prefill(case["q"], out, H, Hkv, dh, case["kc"], case["vc"], ps, case["bt"],
                           case["pos"], case["seq"], tok0, ntok, scale, window)
    torch.cuda.synchronize()
    assert o.attention_tc_error() == 0
    assert torch.allclose(out.float().cpu(), want, **tol(torch.bfloat16))


def test_attention_tc_far_key_and_growing_scores():
    """Head size 128 through the dispatch: one key among 700 carries nearly all the weight
    (a tile's or a page's edge would lose it), and scores that grow along the keys force the
    kernel to move its running maximum and rescale what it has summed."""
    H, Hkv, dh, ps = 8, 2, 128, 16
    for far in (0, 127, 128, 255, 256, 640, 699):
        def crafted(b, K, V, far=far):
            K *= 0.05
            K[far] = 0
            K[far, :, 0] = 30.0
            V[far] = 7.0
        case = paged_case([40], [660], H, Hkv, dh, ps, torch.bfloat16, seed=far, crafted=crafted)
        q = torch.zeros_like(case["q"])
        q[:, 0::dh] = 8.0
        case["q"] = q
        out = torch.zeros_like(q)
        attention_part().paged_attention(q, out, H, Hkv, dh, Cache(case, ps), Ctx(case, False), 1 / math.sqrt(dh), 0)
        sees = case["pos"] >= far
        assert torch.allclose(out[sees].float(), torch.full_like(out[sees], 7.0).float(), atol=0.05), far

    def ramp(b, K, V):
        n = K.shape[0]
        K[:] = 0
        K[:, :, 0] = torch.arange(n, dtype=torch.float32)[:, None] * 0.25     # later keys score higher
    case = paged_case([64], [600], H, Hkv, dh, ps, torch.bfloat16, seed=5, crafted=ramp)
    q = torch.zeros_like(case["q"])
    q[:, 0::dh] = 4.0
    case["q"] = q
    want = attention_ref(case, H, Hkv, dh, 1.0, 0)
    out = torch.zeros_like(q)
    attention_part().paged_attention(q, out, H, Hkv, dh, Cache(case, ps), Ctx(case, False), 1.0, 0)
    assert ops().attention_tc_error() == 0
    assert torch.allclose(out.float().cpu(), want, **tol(torch.bfloat16))


@pytest.mark.parametrize("window", [0, 300])
def test_attention_decode_beyond_the_on_chip_table(window):
    """One decode token 17000 keys into its request (head size 128, pages of 16): more pages
    than the kernel keeps of the block table in shared memory, so the rest comes from global
    memory; with and without key splits."""
    H, Hkv, dh, ps = 4, 1, 128, 16
    case = paged_case([1, 1], [17000, 5], H, Hkv, dh, ps, torch.bfloat16, seed=9)
    scale = 1 / math.sqrt(dh)
    want = attention_ref(case, H, Hkv, dh, scale, window)
    for n_splits in (1, 7):
        out = torch.zeros_like(case["q"])
        ops().attention_flash(case["q"], out, H, Hkv, dh, case["kc"], case["vc"], ps, case["bt"],
                              case["pos"], case["seq"], None, None, scale, window,
                              n_splits=n_splits)
        assert torch.allclose(out.float().cpu(), want, **tol(torch.bfloat16)), n_splits
    assert ops().attention_decode_tma_error() == 0


@pytest.mark.parametrize("H,Hkv,dh,ps", [(8, 2, 64, 16), (5, 1, 128, 8), (16, 1, 64, 32), (4, 4, 128, 64)])
@pytest.mark.parametrize("window,keep", [(0, 0), (130, 0), (140, 5), (300, 200)])
@pytest.mark.parametrize("extra", ["sink", "cap", "bias", "all"])
def test_attention_tc_options(H, Hkv, dh, ps, window, keep, extra):
    """The tcgen05 attention with a sink, kept first keys, bounded scores, a bias by distance and a
    gate, against the generic kernel's float32 arithmetic on the same stored values. P and the
    result are rounded to bfloat16, as in the plain form."""
    case = paged_case([150, 1, 40, 261], [333, 500, 0, 7], H, Hkv, dh, ps, torch.bfloat16, seed=dh + ps)
    T = case["q"].shape[0]
    kw = dict(softcap=2.0 if extra in ("cap", "all") else 0.0, keep_first=keep,
              dist_bias=rnd(70, H, seed=1) if extra in ("bias", "all") else None,
              sinks=rnd(H, seed=2) if extra in ("sink", "all") else None,
              gate=rnd(T, H, seed=3).to(torch.bfloat16) if extra == "all" else None)
    scale, o = dh ** -0.5, ops()
    if keep:
        # what lies between the kept keys and the window of every token of the step has gone back
        for i in range(-(-keep // ps), max(0, 333 - window + 1) // ps):
            case["bt"][0, i] = 0
    t0, nt = attention_part().step_tiles(Ctx(case, False), 128 // (H // Hkv))
    out = torch.full_like(case["q"], 9.0)
    o.attention_tc_prefill(case["q"], out, H, Hkv, dh, case["kc"], case["vc"], ps, case["bt"], case["pos"],
                           case["seq"], t0, nt, scale, window, own_counters=True, **kw)
    want = torch.empty_like(case["q"].float())
    if kw["gate"] is not None:
        kw["gate"] = kw["gate"].float()
    o.attention_generic(case["q"].float(), want, H, Hkv, dh, case["kc"].float(), case["vc"].float(), ps, case["bt"],
                        case["seq"], case["pos"], scale, window, **kw)
    assert o.attention_tc_error() == 0
    assert bool(torch.isfinite(want).all())
    assert torch.allclose(out.float(), want, **tol(torch.bfloat16))


@pytest.mark.parametrize("T,d,ff,E,top", [(127, 64, 32, 1, 1), (128, 72, 40, 1, 1), (129, 136, 264, 1, 1), (257, 200, 104, 2, 1),
                                          (1, 2048, 520, 8, 3), (300, 520, 136, 5, 2), (700, 64, 776, 3, 2), (9, 8, 8, 4, 4)])
@pytest.mark.parametrize("gated,activation", [(True, "silu"), (True, "gelu_tanh"), (False, "relu_squared"), (False, "silu")])
def test_routed_experts_on_tensor_cores(T, d, ff, E, top, gated, activation):
    """Row tiles at and past 128 rows of one expert, column tiles and k-blocks cut short, experts
    without tokens. Hidden rows are bfloat16 (2^-9 each, ff of them in a sum), sums float32."""
    o = ops()
    if activation not in o.PLAIN_ACTIVATIONS or (gated and activation not in o.ACTIVATIONS):
        pytest.skip("not an activation of this form")
    x = rnd(T, d, seed=1).to(torch.bfloat16)
    wr = rnd(E, d, seed=2) * d ** -0.5
    wg, wu = ((rnd(E, ff, d, seed=s) * d ** -0.5).to(torch.bfloat16) for s in (3, 4))
    wd = (rnd(E, d, ff, seed=5) * ff ** -0.5).to(torch.bfloat16)
    got = o.moe_feed_forward(x, wr, None, wg if gated else None, wu, wd, top, activation)
    assert o.moe_error() == 0
    fn = {"silu": torch.nn.functional.silu, "relu_squared": lambda v: torch.relu(v) ** 2, "relu": torch.relu,
          "gelu_tanh": lambda v: torch.nn.functional.gelu(v, approximate="tanh")}[activation]
    z = x.double() @ wr.double().t()
    ids = torch.topk(z, top, -1).indices
    wt = torch.softmax(torch.gather(z, 1, ids), -1)
    want, size = torch.zeros(T, d, dtype=torch.float64, device=DEV), torch.zeros(T, d, dtype=torch.float64, device=DEV)
    for e in range(E):
        row, place = torch.nonzero(ids == e, as_tuple=True)
        xe = x[row].double()
        h = fn(xe @ wu[e].double().t()) if not gated else fn(xe @ wg[e].double().t()) * (xe @ wu[e].double().t())
        want.index_add_(0, row, (h @ wd[e].double().t()) * wt[row, place][:, None])
        size.index_add_(0, row, (h.abs() @ wd[e].double().abs().t()) * wt[row, place][:, None])
    assert ((got.double() - want).abs() <= 2.0 ** -8 * size + 1e-5).all()


@pytest.mark.parametrize("T", [1, 5, 67, 1203])
@pytest.mark.parametrize("H,G,dk,dv,rot,biased,parts", [(16, 4, 128, 128, 64, True, 3), (3, 1, 48, 32, 16, True, 3), (2, 2, 64, 128, 64, False, 3),
                                                        (8, 8, 96, 64, 0, True, 3), (6, 2, 80, 16, 48, True, 2), (5, 1, 256, 64, 256, False, 1)])
def test_projection_rows_the_same_bits_by_either_form(T, H, G, dk, dv, rot, biased, parts):
    """Rows that begin off 16 bytes go a channel a lane: the same bits, with and without keys, values, biases and a rotation."""
    o, ps = ops(), 16
    w, at = H * dk + G * (dk + dv), [H * dk, H * dk + G * dk]
    x = rnd(T, w, seed=dk).to(torch.bfloat16)
    bias = [b.contiguous() if biased else None for b in rnd(w, seed=3).split([at[0], G * dk, G * dv])]
    rope = rnd(T, rot, seed=4) if rot else None
    slots = torch.randperm(T + 9, generator=torch.Generator().manual_seed(1))[:T].to(torch.int32).to(DEV)
    pages, outs = (T + 9 + ps - 1) // ps, []
    for off in (0, 1):
        z = torch.zeros(T, (w + 15) // 8 * 8 + off, dtype=torch.bfloat16, device=DEV)[:, off:w + off]
        z.copy_(x)
        kc, vc = (torch.zeros((pages, G, ps, n), dtype=torch.bfloat16, device=DEV) for n in (dk, dv))
        q, k, v = z[:, :at[0]], z[:, at[0]:at[1]] if parts > 1 else None, z[:, at[1]:] if parts > 2 else None
        o.qkv_bias_rope_cache(q, k, v, H, G if parts > 1 else 0, dk, dv, *bias, rope, rot, False, slots if parts > 1 else None,
                              kc if parts > 1 else None, vc if parts > 2 else None, ps)
        outs.append((z.clone(), kc, vc))
    assert all(torch.equal(a, b) for a, b in zip(*outs))


@pytest.mark.parametrize("T,d", [(5, 136), (300, 72)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_routed_experts_rounded(T, d, dtype):
    """Results in bfloat16 are the float32 ones rounded, with what is added to them, of rows and matrices of either type."""
    o, ff, top, E = ops(), 40, 2, 6
    x = rnd(T, d, seed=1).to(dtype)
    wr = rnd(E, d, seed=2) * d ** -0.5
    wg, wu = ((rnd(E, ff, d, seed=s) * d ** -0.5).to(dtype) for s in (3, 4))
    wd = (rnd(E, d, ff, seed=5) * ff ** -0.5).to(dtype)
    run = lambda **kw: o.moe_feed_forward(x, wr, None, wg, wu, wd, top, "silu", rnd(T, d, seed=6),       # noqa: E731
                                          beside=rnd(T, d, seed=7).to(torch.bfloat16), **kw)
    assert torch.equal(run(out_dtype=torch.bfloat16), run().to(torch.bfloat16))


@pytest.mark.parametrize("T,E,identity,top", [(9, 4, 0, 2), (9, 4, 4, 3), (200, 4, 0, 2), (200, 4, 4, 3)])
@pytest.mark.parametrize("strided", [False, True])
def test_routed_experts_of_strided_rows_and_identities(T, E, identity, top, strided):
    """Rows of x with a stride of their own and router outputs that stand for the row itself, with few rows
    an expert (gathered) and many (copied in place order; identities have no place there)."""
    o, d, ff = ops(), 136, 104
    assert (T * top >= o.MOE_GATHER_ROWS * E) == (T == 200)
    x = rnd(T, d + 24, seed=1).to(torch.bfloat16)[:, 8:d + 8] if strided else rnd(T, d, seed=1).to(torch.bfloat16)
    wr = rnd(E + identity, d, seed=2) * d ** -0.5
    wg, wu = ((rnd(E, ff, d, seed=s) * d ** -0.5).to(torch.bfloat16) for s in (3, 4))
    wd = (rnd(E, d, ff, seed=5) * ff ** -0.5).to(torch.bfloat16)
    got = o.moe_feed_forward(x, wr, None, wg, wu, wd, top, "silu", scores="all", identity=identity)
    assert o.moe_error() == 0
    p = torch.softmax(x.double() @ wr.double().t(), -1)
    ids = torch.topk(p, top, -1).indices
    wt = torch.gather(p, 1, ids)
    wt = wt / wt.sum(-1, keepdim=True)
    want, size = torch.zeros(T, d, dtype=torch.float64, device=DEV), torch.zeros(T, d, dtype=torch.float64, device=DEV)
    for e in range(E + identity):
        row, place = torch.nonzero(ids == e, as_tuple=True)
        xe, we = x[row].double(), wt[row, place][:, None]
        if e >= E:
            want.index_add_(0, row, xe * we)
            continue
        h = torch.nn.functional.silu(xe @ wg[e].double().t()) * (xe @ wu[e].double().t())
        want.index_add_(0, row, (h @ wd[e].double().t()) * we)
        size.index_add_(0, row, (h.abs() @ wd[e].double().abs().t()) * we)
    assert not identity or (ids >= E).any()
    # hidden rows are rounded to bfloat16 (2^-9 each); the rest is float32
    assert ((got.double() - want).abs() <= 2.0 ** -8 * size + 1e-5).all()


def test_routed_experts_activation_in_32_bits():
    """SiLU of products far below zero. The products are sums of two exact numbers, so that the hidden rows
    show the activation alone: within 2^-21 (the exponential's 2 units in the last place, a sum, a
    product and a division of half a unit each: 2^-21.2) and one rounding to bfloat16 of the value in 64 bits."""
    o, d = ops(), 256
    a = torch.cat([torch.arange(-88, -64, 0.5), torch.arange(-64, -32, 0.25), torch.arange(-32, -16, 0.125),
                   torch.arange(-16, 16, 0.25)])
    x = torch.zeros(a.numel(), d)
    x[:, 0], x[:, 1] = a, 1.0
    wg, wu = torch.zeros(1, d, d), torch.zeros(1, d, d)
    wg[0, :, 0], wg[0, :, 1], wu[0, :, 1] = 1.0, torch.arange(d) / 8192.0, 1.0
    x, wg, wu, wd = (t.to(torch.bfloat16).to(DEV) for t in (x, wg, wu, torch.eye(d)[None]))
    got = o.moe_feed_forward(x, torch.zeros(1, d, device=DEV), None, wg, wu, wd, 1, "silu").double()
    z = x.double() @ wg[0].double().t()
    want = z / (1.0 + torch.exp(-z))
    half = torch.exp2(torch.floor(torch.log2(want.abs())) - 8)           # half of what bfloat16 is spaced by
    assert o.moe_error() == 0 and torch.equal(got, got.to(torch.bfloat16).double())
    assert ((got - want).abs() <= half + 2.0 ** -21 * want.abs()).all()
    # a product that overflows to infinity keeps it, one to the other side is no number (0 x infinity)
    x, wg = torch.zeros(2, d, dtype=x.dtype, device=DEV), torch.zeros_like(wg)
    x[:, 1], x[0, 0], x[1, 0], wg[0, 0, 0] = 1.0, 3e38, -3e38, 2.0
    got = o.moe_feed_forward(x, torch.zeros(1, d, device=DEV), None, wg, wu, wd, 1, "silu")
    assert got[0, 0] == float("inf") and bool(torch.isnan(got[1, 0]))


@pytest.mark.parametrize("dk,dv,rot,act", [(64, 8, 0, 0), (64, 128, 32, 1), (128, 136, 128, 0), (128, 256, 64, 1)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_retention_by_tiled_chunks(dk, dv, rot, act, dtype):
    """Heads the tensor-core kernels take, requests that end before, on and after a chunk, against
    the recurrence in 64 bits: sums of at most dk + 64 float32 terms behind at most ten chunks."""
    o, H, lens = ops(), 3, [1, 63, 64, 65, 200, 577]
    T, B = sum(lens), len(lens)
    z = (rnd(T, H * (2 * dk + dv), seed=dk + dv) * 0.5).to(dtype)
    q, k, v = z[:, :H * dk], z[:, H * dk:2 * H * dk], z[:, 2 * H * dk:]
    decay = torch.tensor([0.5, 0.97, 1.0], device=DEV)
    rope = torch.randn(T, rot, device=DEV) if rot else None
    state = rnd(B + 2, H, dk, dv, seed=1)
    before, slots = state.clone(), [3, 0, 5, 1, 7, 2]
    starts = [0]
    for n in lens:
        starts.append(starts[-1] + n)
    C, t0, nt, first = o.retention_chunk_tokens(), [], [], []
    for s, n in zip(starts, lens):
        first.append(len(t0))
        t0 += range(s, s + n, C)
        nt += [min(C, n - a) for a in range(0, n, C)]
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)       # noqa: E731
    out = torch.full((T, H * dv), float("nan"), device=DEV)
    o.retention_chunked(q, k, v, out, B, H, dk, dv, decay, dk ** -0.5, rope, rot, i32(starts), i32(slots), state,
                        i32(t0), i32(nt), i32(first), act=act)

    def taken(x, w, turned):
        x = x.double().view(T, H, w)
        if act:
            x = torch.nn.functional.silu(x)
        if not turned or not rot:
            return x
        c, s = rope.double()[:, None, :rot // 2], rope.double()[:, None, rot // 2:]
        a, b = x[..., :rot // 2], x[..., rot // 2:rot]
        return torch.cat([a * c - b * s, b * c + a * s, x[..., rot:]], -1)
    qq, kk, vv = taken(q, dk, True), taken(k, dk, True) * dk ** -0.5, taken(v, dv, False)
    for b, n in enumerate(lens):
        S = before[slots[b]].double()
        want = torch.empty(n, H, dv, dtype=torch.float64, device=DEV)
        for i in range(n):
            t = starts[b] + i
            S = decay.double()[:, None, None] * S + kk[t][:, :, None] * vv[t][:, None]
            want[i] = torch.einsum("hkv,hk->hv", S, qq[t])
        got = out[starts[b]:starts[b + 1]].view(n, H, dv).double()
        assert (got - want).norm() <= 3e-6 * want.norm() and (state[slots[b]].double() - S).norm() <= 3e-6 * S.norm()
    untouched = [i for i in range(B + 2) if i not in slots]
    assert torch.equal(state[untouched], before[untouched])


@pytest.mark.parametrize("lens", [[0, 70, 0, 0, 64, 0], [130, 0, 1]])
def test_retention_by_tiled_chunks_beside_empty_requests(lens):
    """Requests without tokens between others: the others' outputs and states, the same bits; theirs stay."""
    o, H, dk, dv = ops(), 2, 64, 128
    C, z = o.retention_chunk_tokens(), rnd(sum(lens), H * (2 * dk + dv), seed=5) * 0.5
    state = rnd(len(lens), H, dk, dv, seed=1)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)       # noqa: E731

    def run(lens, slots):
        starts, t0, nt, first = [0], [], [], []
        for n in lens:
            first.append(len(t0))
            t0 += range(starts[-1], starts[-1] + n, C)
            nt += [min(C, n - a) for a in range(0, n, C)]
            starts.append(starts[-1] + n)
        out, s = torch.full((sum(lens), H * dv), float("nan"), device=DEV), state.clone()
        o.retention_chunked(z[:, :H * dk], z[:, H * dk:2 * H * dk], z[:, 2 * H * dk:], out, len(lens), H, dk, dv,
                            torch.tensor([0.9, 0.99], device=DEV), dk ** -0.5, None, 0, i32(starts), i32(slots), s,
                            i32(t0), i32(nt), i32(first))
        return out, s
    full = [i for i, n in enumerate(lens) if n]
    got, want = run(lens, list(range(len(lens)))), run([lens[i] for i in full], full)
    assert bool(torch.isfinite(got[0]).all()) and torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
    assert torch.equal(got[1][[i for i, n in enumerate(lens) if not n]], state[[i for i, n in enumerate(lens) if not n]])


@pytest.mark.parametrize("dk,dv", [(64, 136), (128, 256)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_retention_by_tiled_chunks_looks_forward_only(dk, dv, dtype):
    """A value, key or query that is not finite at a token leaves every output before it, and the other
    channels of the value, as they are without it."""
    o, H, n = ops(), 2, 150
    z = (rnd(n, H * (2 * dk + dv), seed=dk + dv) * 0.5).to(dtype)
    C = o.retention_chunk_tokens()
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)       # noqa: E731
    nt = [min(C, n - a) for a in range(0, n, C)]

    def run(z):
        out, state = torch.empty(n, H * dv, device=DEV), torch.zeros(1, H, dk, dv, device=DEV)
        o.retention_chunked(z[:, :H * dk], z[:, H * dk:2 * H * dk], z[:, 2 * H * dk:], out, 1, H, dk, dv,
                            torch.tensor([0.9, 0.99], device=DEV), dk ** -0.5, None, 0, i32([0, n]), i32([0]), state,
                            i32(list(range(0, n, C))), i32(nt), i32([0]))
        return out
    clean = run(z)
    assert bool(torch.isfinite(clean).all())
    for t in (0, 1, 6, 7, 37, 63, 64, 75, 149):
        for bad in (float("nan"), float("inf"), float("-inf")):
            for col in (3, H * dk + 5, 2 * H * dk + 9):                  # a query, a key and a value of head 0
                y = z.clone()
                y[t, col] = bad
                got = run(y)
                assert torch.equal(got[:t], clean[:t]), (t, bad, col)
                assert not bool(torch.isfinite(got[t, :dv]).all()) and torch.equal(got[:, dv:], clean[:, dv:])
                if col >= 2 * H * dk:
                    others = [c for c in range(dv) if c != 9]
                    assert torch.equal(got[:, others], clean[:, others]), (t, bad)


def retention_of_one(z, H, dk, dv, decay, k_scale, state, act=0):
    """One request through the chunked retention, its rows [q, k, v]: outputs [n, H, dv]; `state` [1, H, dk, dv] moves on."""
    o, n = ops(), z.shape[0]
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)       # noqa: E731
    C, out = o.retention_chunk_tokens(), torch.full((n, H * dv), float("nan"), device=DEV)
    o.retention_chunked(z[:, :H * dk], z[:, H * dk:2 * H * dk], z[:, 2 * H * dk:], out, 1, H, dk, dv,
                        torch.tensor(decay, device=DEV), k_scale, None, 0, i32([0, n]), i32([0]), state,
                        i32(list(range(0, n, C))), i32([min(C, n - a) for a in range(0, n, C)]), i32([0]), act=act)
    assert o.retention_error() == 0
    return out.view(n, H, dv)


@pytest.mark.parametrize("dk,dv", [(64, 136), (64, 256), (128, 136), (128, 256), (128, 384)])
@pytest.mark.parametrize("dtype,act", [(torch.float32, 0), (torch.bfloat16, 0), (torch.bfloat16, 1)])
def test_retention_by_chunks_of_two_slices_a_block(dk, dv, dtype, act):
    """Steps whose blocks take two slices of 128 value channels, the last cut or alone, against the recurrence in 64 bits; the bits
    of a step so short that they take one. What is not finite in a second slice stays in its channel."""
    H, n, decay = 4, 1300, [0.5, 0.9, 0.97, 1.0]
    slices, sms = (dv + 127) // 128, torch.cuda.get_device_properties(0).multi_processor_count
    assert (n + 63) // 64 * H * slices > sms >= 3 * H * slices           # two slices a block here, one in the short step
    z = (rnd(n, H * (2 * dk + dv), seed=dk + dv) * 0.5).to(dtype)
    start = rnd(1, H, dk, dv, seed=1)
    state, short = start.clone(), start.clone()
    got = retention_of_one(z, H, dk, dv, decay, dk ** -0.5, state, act)
    assert torch.equal(retention_of_one(z[:150], H, dk, dv, decay, dk ** -0.5, short, act), got[:150])
    q, k, v = (x.double().view(n, H, -1) for x in z.split([H * dk, H * dk, H * dv], 1))
    if act:
        q, k, v = (torch.nn.functional.silu(x) for x in (q, k, v))
    S, want = start[0].double(), torch.empty(n, H, dv, dtype=torch.float64, device=DEV)
    g = torch.tensor(decay, device=DEV).double()[:, None, None]
    for t in range(n):
        S = g * S + (k[t] * dk ** -0.5)[:, :, None] * v[t][:, None]
        want[t] = torch.einsum("hkv,hk->hv", S, q[t])
    # sums of dk + 64 float32 terms behind 21 chunks, and a chunk's powers of the decay by up to 64 products
    for a in range(0, dv, 128):                          # a slice for itself, so that none hides behind another
        b = min(dv, a + 128)
        assert (got[:, :, a:b].double() - want[:, :, a:b]).norm() <= 3e-6 * want[:, :, a:b].norm()
        assert (state[0, :, :, a:b].double() - S[:, :, a:b]).norm() <= 3e-6 * S[:, :, a:b].norm()
    for t in (0, 70, 1299):
        for bad in (float("nan"), float("inf")):
            y = z.clone()
            y[t, 2 * H * dk + dv + 130] = bad            # head 1
            odd = retention_of_one(y, H, dk, dv, decay, dk ** -0.5, start.clone(), act)
            others = torch.ones(H, dv, dtype=torch.bool, device=DEV)
            others[1, 130] = False
            assert torch.equal(odd[:t], got[:t]) and torch.equal(odd[:, others], got[:, others])
            assert not bool(torch.isfinite(odd[t, 1, 130]))
    if dtype == torch.float32:                           # too large for its parts: its slice of its head takes plain sums
        y = z.clone()
        y[70, 2 * H * dk + dv + 130] = 1e32
        odd = retention_of_one(y, H, dk, dv, decay, dk ** -0.5, start.clone(), act)
        assert torch.equal(odd[:70], got[:70]) and torch.equal(odd[:, [0, 2, 3]], got[:, [0, 2, 3]]) and torch.equal(odd[:, 1, :128], got[:, 1, :128])
        score = (q[:, 1] @ (k[70, 1] * dk ** -0.5)) * g[1, 0, 0] ** torch.arange(-70, n - 70, device=DEV)
        assert bool(((odd[70:, 1, 130].double() - want[70:, 1, 130] - 1e32 * score[70:]).abs() <= 1e32 * 1e-5 * score[70:].abs() + 1e26).all())


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_retention_by_chunks_of_large_scores(dtype):
    """A score near the end of the range whose second half of channels is past it alone: the sum over all channels is
    finite in the order of the channels, and so is its share of the output. Rows before are as they are without it."""
    H, dk, dv, n, key, query = 2, 128, 136, 100, 70, 75
    z = (rnd(n, H * (2 * dk + dv), seed=4) * 0.5).to(dtype)
    at = [0, 64, 65]
    for t in range(n):                                   # the three channels are the two tokens' own, in head 0
        z[t, at], z[t, [dk * H + c for c in at]] = 0.0, 0.0
    clean = retention_of_one(z, H, dk, dv, [1.0, 0.9], 1.0, torch.zeros(1, H, dk, dv, device=DEV))
    z[query, :dk], z[key, H * dk:H * dk + dk], z[key, 2 * H * dk:2 * H * dk + dv] = 0.0, 0.0, 1e-30
    for i, c in enumerate(at):
        z[query, c], z[key, H * dk + c] = 1.7e19, -1.7e19 if i == 0 else 1.7e19
    got = retention_of_one(z, H, dk, dv, [1.0, 0.9], 1.0, torch.zeros(1, H, dk, dv, device=DEV))
    assert torch.equal(got[:key], clean[:key]) and torch.equal(got[:, 1], clean[:, 1])
    q, k, v = z[query, :dk].double(), z[key, H * dk:H * dk + dk].double(), z[key, 2 * H * dk:2 * H * dk + dv].double()
    want = (q @ k) * v                                   # 2.9e8; the channels meet no other key
    assert bool(((got[query, 0].double() - want).abs() <= 1e-6 * want).all()), (got[query, 0, :4], want[:4])


@pytest.mark.parametrize("dk,dv", [(64, 64), (128, 136)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("qs,ks,vs,ss", [(1.0, 1.0, 1e-36, 1e-36), (1e-36, 1.0, 1.0, 1.0), (1.0, 1e-36, 1.0, 1e-36), (1e-20, 1e-16, 1.0, 1e-16),
                                         (1e33, 1e-30, 1.0, 1e-30), (1e-30, 1e33, 1.0, 1e30), (1.0, 1e-30, 1e33, 1e5), (1e-30, 1.0, 1.0, 1e34)])
def test_retention_by_chunks_of_small_and_large_numbers(dk, dv, dtype, qs, ks, vs, ss):
    """Numbers whose lower parts have no bfloat16 number of their size, scores of such a size, and numbers past those that
    the parts are scaled for, against the recurrence in 64 bits: the bound of ordinary numbers."""
    H, n, decay = 2, 130, [0.9, 1.0]
    z = rnd(n, H * (2 * dk + dv), seed=dk).to(dtype)
    z[:, :H * dk] *= qs
    z[:, H * dk:2 * H * dk] *= ks
    z[:, 2 * H * dk:] *= vs
    state = rnd(1, H, dk, dv, seed=1) * ss
    S, want = state[0].double(), torch.empty(n, H, dv, dtype=torch.float64, device=DEV)
    q, k, v = (x.double().view(n, H, -1) for x in z.split([H * dk, H * dk, H * dv], 1))
    for t in range(n):
        S = torch.tensor(decay, dtype=torch.float64, device=DEV)[:, None, None] * S + k[t][:, :, None] * v[t][:, None]
        want[t] = torch.einsum("hkv,hk->hv", S, q[t])
    got = retention_of_one(z, H, dk, dv, decay, 1.0, state).double()
    for h in range(H):
        assert (got[:, h] - want[:, h]).norm() <= 1e-6 * want[:, h].norm()
        # a state that is mostly the one before, n powers of the decay later, has a rounding of each of them on top
        assert (state[0, h].double() - S[h]).norm() <= (1e-6 + n * 2.0 ** -24) * S[h].norm()


def best_time(run):
    best = float("inf")
    for _ in range(5):
        t = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
        t[0].record()
        run()
        t[1].record()
        torch.cuda.synchronize()
        best = min(best, t[0].elapsed_time(t[1]))
    return best


def test_chunked_kernels_of_no_numbers_at_a_time_of_their_kind(monkeypatch):
    """Rows of NaN through retention and the selective scan by chunks: plain sums of sixteen rows a thread take seven to eight times
    as long as a finite call, a sum a thread out of global memory took fifteen and more."""
    z = rnd(4096, 16 * 512, seed=1).to(torch.bfloat16)
    state = torch.zeros(1, 16, 128, 256, device=DEV)
    run = lambda z: retention_of_one(z, 16, 128, 256, [0.9] * 16, 1.0, state.zero_())      # noqa: E731
    bad = torch.full_like(z, float("nan"))
    assert bool(torch.isnan(run(bad)).all()) and best_time(lambda: run(bad)) <= 11 * best_time(lambda: run(z))
    xbc, dt_raw, a_log = rnd(2048, 64 * 64 + 16 * 128, seed=1), rnd(2048, 64, seed=3).to(torch.bfloat16), torch.zeros(64, device=DEV)
    run = lambda x: chunked_scan(ops(), monkeypatch, x, dt_raw, a_log, 64, 8, 128, 64)[0]      # noqa: E731
    bad = torch.full_like(xbc, float("nan"))
    assert bool(torch.isnan(run(bad)).all()) and best_time(lambda: run(bad)) <= 11 * best_time(lambda: run(xbc))


def scan_in_64_bits(xbc, dt_raw, a_log, d, H, G, N, P):
    T = xbc.shape[0]
    x, B, C = (z.double() for z in xbc.split([H * P, G * N, G * N], 1))
    B, C = (z.view(T, G, N).repeat_interleave(H // G, 1) for z in (B, C))
    dt, S = torch.nn.functional.softplus(dt_raw.double()), torch.zeros(H, N, P, dtype=torch.float64, device=DEV)
    want = torch.empty(T, H, P, dtype=torch.float64, device=DEV)
    for t in range(T):
        S = torch.exp(-torch.exp(a_log.double()) * dt[t])[:, None, None] * S + \
            (dt[t][:, None] * B[t])[:, :, None] * x[t].view(H, 1, P)
        want[t] = torch.einsum("hn,hnp->hp", C[t], S) + (0.0 if d is None else d.double()[:, None] * x[t].view(H, P))
    return want, S


def chunked_scan(o, monkeypatch, xbc, dt_raw, a_log, H, G, N, P, chunks=True, d=None):
    """One request through the selective scan by chunks or in order (None: as the rule has it beyond the
    shortest steps): outputs and state."""
    T = xbc.shape[0]
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)       # noqa: E731
    y, state = torch.empty(T, H * P, device=DEV), torch.zeros(1, H * N * P, device=DEV)
    monkeypatch.setattr(o, "SSD_MIN_TOKENS", 1 << 30 if chunks is False else 1)
    launches = o.LAUNCHES[0]
    o.selective_scan(xbc, dt_raw, None, a_log, d, y, 1, H, G, N, P, i32([0, T]), i32([0]), state, 0)
    assert chunks is None or o.LAUNCHES[0] == launches + (4 if chunks else 1)
    return y, state


@pytest.mark.parametrize("H,G,N,P,T", [(6, 2, 64, 64, 200), (40, 2, 128, 64, 65), (40, 2, 128, 64, 1500), (5, 1, 128, 128, 190),
                                       (12, 1, 64, 64, 64), (17, 1, 64, 128, 257)])
def test_selective_scan_by_chunks_heads_a_block(H, G, N, P, T, monkeypatch):
    """Groups whose heads fill blocks and pairs of 128 channels or do not, whole and cut chunks, against the
    recurrence in 64 bits: sums of N + 64 float32 terms behind at most T / 64 chunks."""
    o = ops()
    xbc, dt_raw = rnd(T, H * P + 2 * G * N, seed=N + T), rnd(T, H, seed=3).to(torch.bfloat16)
    a_log = torch.linspace(-2.0, 1.0, H, device=DEV)
    y, state = chunked_scan(o, monkeypatch, xbc, dt_raw, a_log, H, G, N, P)
    x, B, C = (z.double() for z in xbc.split([H * P, G * N, G * N], 1))
    B, C = (z.view(T, G, N).repeat_interleave(H // G, 1) for z in (B, C))
    dt, S = torch.nn.functional.softplus(dt_raw.double()), torch.zeros(H, N, P, dtype=torch.float64, device=DEV)
    want = torch.empty(T, H, P, dtype=torch.float64, device=DEV)
    for t in range(T):
        S = torch.exp(-torch.exp(a_log.double()) * dt[t])[:, None, None] * S + \
            (dt[t][:, None] * B[t])[:, :, None] * x[t].view(H, 1, P)
        want[t] = torch.einsum("hn,hnp->hp", C[t], S)
    assert (y.view(T, H, P).double() - want).norm() <= 1e-6 * want.norm()
    assert (state.view(H, N, P).double() - S).norm() <= 1e-6 * S.norm()
    assert o.ssd_error() == 0


@pytest.mark.parametrize("N", [64, 128])
@pytest.mark.parametrize("P", [64, 128])
def test_selective_scan_by_chunks_pairs_in_turn(N, P, monkeypatch):
    """Blocks of five heads, which are three turns of 128 channels (the last half full) or five, with x beside the sums,
    against the recurrence in 64 bits; what is not finite in a last turn stays there."""
    o, H, G, T = ops(), 40, 2, 1500
    # 24 chunks: five heads a block are 192 blocks, ten would be 96, fewer than the multiprocessors there are
    assert 24 * 8 >= torch.cuda.get_device_properties(0).multi_processor_count > 24 * 4
    xbc, dt_raw = rnd(T, H * P + 2 * G * N, seed=N + P), rnd(T, H, seed=3).to(torch.bfloat16)
    a_log, d = torch.linspace(-2.0, 1.0, H, device=DEV), rnd(H, seed=5)
    run = lambda x: chunked_scan(o, monkeypatch, x, dt_raw, a_log, H, G, N, P, d=d)      # noqa: E731
    y, state = run(xbc)
    want, S = scan_in_64_bits(xbc, dt_raw, a_log, d, H, G, N, P)
    # for each head, so that none hides behind the others: sums of N + 64 float32 terms behind at most 24 chunks
    assert bool(((y.view(T, H, P).double() - want).norm(dim=(0, 2)) <= 1e-6 * want.norm(dim=(0, 2))).all())
    assert bool(((state.view(H, N, P).double() - S).norm(dim=(1, 2)) <= 1e-6 * S.norm(dim=(1, 2))).all())
    for t, head in ((0, 4), (70, 3), (1499, 39)):
        for bad in (float("nan"), float("inf")):
            z = xbc.clone()
            z[t, head * P + 9] = bad
            got, _ = run(z)
            others = [c for c in range(H * P) if c != head * P + 9]
            assert torch.equal(got[:t], y[:t]) and torch.equal(got[:, others], y[:, others])
            assert not bool(torch.isfinite(got[t, head * P + 9]))
    assert o.ssd_error() == 0


@pytest.mark.parametrize("H,G,N,P", [(64, 8, 128, 64), (3, 1, 64, 64), (2, 1, 128, 128)])
def test_selective_scan_by_chunks_looks_forward_only(H, G, N, P, monkeypatch):
    """A number that is not finite at a token leaves every output before it as it is without it; one in x
    leaves the other channels' too. Two heads a block and one."""
    o, T = ops(), 200
    xbc, dt_raw = rnd(T, H * P + 2 * G * N, seed=N + P), rnd(T, H, seed=3).to(torch.bfloat16)
    a_log = torch.linspace(-3.0, 1.0, H, device=DEV)
    clean, _ = chunked_scan(o, monkeypatch, xbc, dt_raw, a_log, H, G, N, P)
    assert bool(torch.isfinite(clean).all())
    for t in (0, 1, 14, 15, 40, 63, 64, 100, 199):
        for bad in (float("nan"), float("inf"), float("-inf")):
            for col in (9, H * P + 5, H * P + G * N + 7):                # of x, of B and of C
                y = xbc.clone()
                y[t, col] = bad
                got, _ = chunked_scan(o, monkeypatch, y, dt_raw, a_log, H, G, N, P)
                assert torch.equal(got[:t], clean[:t]), (t, bad, col)
                assert not bool(torch.isfinite(got[t, :P]).all())
                if col == 9:
                    others = [c for c in range(H * P) if c != 9]
                    assert torch.equal(got[:, others], clean[:, others]), (t, bad)
        y = dt_raw.clone()
        y[t, 0] = float("nan")
        got, _ = chunked_scan(o, monkeypatch, xbc, y, a_log, H, G, N, P)
        assert torch.equal(got[:t], clean[:t]) and torch.equal(got[:, P:], clean[:, P:])
        assert bool(torch.isnan(got[t:, :P]).all())


@pytest.mark.parametrize("N,P", [(64, 64), (128, 64), (64, 128), (128, 128)])
@pytest.mark.parametrize("xs,bs,cs", [(1e-36, 1.0, 1.0), (1.0, 1e-36, 1.0), (1.0, 1.0, 1e-36), (1.0, 1e-20, 1e-16), (1e33, 1e-20, 1.0),
                                      (1e-20, 1e33, 1.0), (1e-20, 1.0, 1e33)])
def test_selective_scan_by_chunks_of_small_and_large_numbers(N, P, xs, bs, cs, monkeypatch):
    """Numbers whose lower parts have no bfloat16 number of their size, and numbers past those that the parts are scaled
    for, in x, B and C and so in the states, against the recurrence in 64 bits: the bound of ordinary numbers."""
    H, T = 3, 150
    xbc, dt_raw = rnd(T, H * P + 2 * N, seed=N + P), rnd(T, H, seed=3).to(torch.bfloat16)
    for at, size, scale in ((0, H * P, xs), (H * P, N, bs), (H * P + N, N, cs)):
        xbc[:, at:at + size] *= scale
    a_log = torch.linspace(-3.0, 0.0, H, device=DEV)
    want, S = scan_in_64_bits(xbc, dt_raw, a_log, None, H, 1, N, P)
    y, state = chunked_scan(ops(), monkeypatch, xbc, dt_raw, a_log, H, 1, N, P)
    assert ops().ssd_error() == 0
    y, state = y.view(T, H, P).double(), state.view(H, N, P).double()
    for h in range(H):
        assert (y[:, h] - want[:, h]).norm() <= 1e-6 * want[:, h].norm() and (state[h] - S[h]).norm() <= 1e-6 * S[h].norm()


@pytest.mark.parametrize("N,P", [(64, 64), (128, 64), (64, 128), (128, 128)])
def test_selective_scan_by_chunks_of_large_factors(N, P, monkeypatch):
    """B, C, dt, D and x whose product is finite though C . B times dt, or with D on top, is past the range: the walk's result.
    Rows before are as they are without it, and so is the other head."""
    o, H, T, key, query, diag = ops(), 2, 100, 70, 73, 80
    xbc, dt_raw = rnd(T, H * P + 2 * N, seed=N + P), rnd(T, H, seed=3).to(torch.bfloat16)
    a_log, d = torch.full((H,), -6.0, device=DEV), torch.tensor([3.3e38, 1.0], device=DEV)
    b, c = H * P, H * P + N
    xbc[:, b] = xbc[:, c] = xbc[:, b + 1] = xbc[:, c + 1] = 0.0
    xbc[:, :P] = 1e-30
    y0, _ = chunked_scan(o, monkeypatch, xbc, dt_raw, a_log, H, 1, N, P, d=d)
    for t, lane, small in ((key, 0, 1e19), (query, 0, 1e19), (diag, 1, 6e18)):
        if t != query:
            xbc[t, b:b + N] = 0.0
            xbc[t, b + lane] = small
        if t != key:
            xbc[t, c:c + N] = 0.0
            xbc[t, c + lane] = small
    dt_raw[key, 0], dt_raw[diag, 0] = 10.0, 0.5
    args = (o, monkeypatch, xbc, dt_raw, a_log, H, 1, N, P)
    got, state = chunked_scan(*args, d=d)
    want, state2 = chunked_scan(*args, chunks=False, d=d)
    assert bool(torch.isfinite(want).all()) and want[query, 0] > 1e9 and want[diag, 0] > 3.6e8
    assert bool(((got - want).abs() <= 1e-5 * want.abs())[[query, diag], :P].all()), (got[query, :3], want[query, :3])
    assert torch.equal(got[:key], y0[:key]) and (state - state2).norm() <= 6e-6 * state2.norm()
    assert bool(((got - want)[:, P:].norm(dim=1) <= 1e-4 * want[:, P:].norm(dim=1)).all()) and o.ssd_error() == 0


@pytest.mark.parametrize("H,G,N,P", [(6, 3, 128, 64), (3, 1, 64, 128)])
def test_selective_scan_by_chunks_with_decays_of_zero(H, G, N, P, monkeypatch):
    """Heads whose state is gone after a token (exp(A_log) up to infinity in 32 bits): what the walk in order
    gives, within the rounding of sums of at most N + 64 float32 terms."""
    o, T = ops(), 300
    xbc, dt_raw = rnd(T, H * P + 2 * G * N, seed=N + P), rnd(T, H, seed=3).to(torch.bfloat16)
    a_log = torch.linspace(60.0, 100.0, H, device=DEV)
    a_log[0] = 0.0
    got, state = chunked_scan(o, monkeypatch, xbc, dt_raw, a_log, H, G, N, P)
    want, state2 = chunked_scan(o, monkeypatch, xbc, dt_raw, a_log, H, G, N, P, chunks=False)
    assert bool(torch.isfinite(want).all())
    assert (got - want).norm() <= 6e-6 * want.norm() and (state - state2).norm() <= 6e-6 * state2.norm()
    assert ((got - want).abs() <= 1e-4 * want.abs().clamp(min=1.0)).all()


@pytest.mark.parametrize("lens", [[0, 70, 0, 0, 64, 0], [130, 0, 1]])
def test_selective_scan_by_chunks_beside_empty_requests(lens, monkeypatch):
    """Requests without tokens between others: the others' outputs and states, the same bits; theirs stay."""
    o, H, G, N, P, T = ops(), 4, 2, 64, 64, sum(lens)
    xbc, dt_raw = rnd(T, H * P + 2 * G * N, seed=1), rnd(T, H, seed=3).to(torch.bfloat16)
    state = rnd(len(lens), H * N * P, seed=6)
    monkeypatch.setattr(o, "SSD_MIN_TOKENS", 1)
    monkeypatch.setattr(o, "SSD_TOKENS_A_REQUEST", 1)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)       # noqa: E731

    def run(lens, slots):
        starts = [0]
        for n in lens:
            starts.append(starts[-1] + n)
        y, s = torch.full((T, H * P), float("nan"), device=DEV), state.clone()
        launches = o.LAUNCHES[0]
        o.selective_scan(xbc, dt_raw, None, torch.linspace(-3.0, 1.0, H, device=DEV), None, y, len(lens), H, G, N, P,
                         i32(starts), i32(slots), s, 0)
        assert o.LAUNCHES[0] == launches + 4
        return y, s
    full = [i for i, n in enumerate(lens) if n]
    got, want = run(lens, list(range(len(lens)))), run([lens[i] for i in full], full)
    assert bool(torch.isfinite(got[0]).all()) and torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])


def test_selective_scan_by_chunks_takes_a_bounded_workspace():
    """16000 tokens of 64 heads of 64 x 128 (a state's size a chunk and head: 525 MB) run in groups of heads
    over at most 256 MB beside the result."""
    o, T, H, G, N, P = ops(), 16000, 64, 8, 128, 64
    xbc, dt_raw = torch.zeros(T, H * P + 2 * G * N, device=DEV), torch.zeros(T, H, dtype=torch.bfloat16, device=DEV)
    y, state, i32 = torch.empty(T, H * P, device=DEV), torch.zeros(1, H * N * P, device=DEV), torch.int32
    torch.cuda.synchronize()
    torch.cuda.reset_peak_memory_stats()
    before = torch.cuda.memory_allocated()
    o.selective_scan(xbc, dt_raw, None, torch.zeros(H, device=DEV), None, y, 1, H, G, N, P,
                     torch.tensor([0, T], dtype=i32, device=DEV), torch.tensor([0], dtype=i32, device=DEV), state, 0)
    torch.cuda.synchronize()
    assert torch.cuda.max_memory_allocated() - before <= (256 << 20) + (1 << 20)
    assert not y.any() and not state.any()


@pytest.mark.parametrize("H,G,N,P", [(24, 4, 128, 64), (3, 1, 128, 64), (5, 1, 64, 128)])
def test_selective_scan_by_chunks_in_groups_of_heads(H, G, N, P, monkeypatch):
    """Heads in groups of every size, down to one, give the bits of all at once; none at all walks."""
    o, T = ops(), 700
    xbc, dt_raw = rnd(T, H * P + 2 * G * N, seed=N + P), rnd(T, H, seed=3).to(torch.bfloat16)
    a_log = torch.linspace(-3.0, 1.0, H, device=DEV)
    y, state = chunked_scan(o, monkeypatch, xbc, dt_raw, a_log, H, G, N, P)
    a_head = 4 * (T // 64 + 1) * (N * P + 3 * 64 + 4)
    for heads in sorted({1, 2, 3, H // 2 + 1} - {H}):
        monkeypatch.setattr(o, "SSD_WORKSPACE_BYTES", heads * a_head)
        launches = o.LAUNCHES[0]
        y2, state2 = chunked_scan(o, monkeypatch, xbc, dt_raw, a_log, H, G, N, P, chunks=None)
        assert (o.LAUNCHES[0] - launches) % 4 == 0 and o.LAUNCHES[0] - launches > 4
        assert torch.equal(y, y2) and torch.equal(state, state2)
    monkeypatch.setattr(o, "SSD_WORKSPACE_BYTES", 1000)
    launches = o.LAUNCHES[0]
    chunked_scan(o, monkeypatch, xbc, dt_raw, a_log, H, G, N, P, chunks=None)
    assert o.LAUNCHES[0] == launches + 1


@pytest.mark.parametrize("H,G,most,at_once", [(64, 8, 22, 16), (64, 8, 40, 32), (48, 2, 30, 24), (6, 2, 4, 3)])
def test_selective_scan_by_chunks_in_blocks_of_heads_at_a_time(H, G, most, at_once, monkeypatch):
    """Blocks of several heads and a workspace for a part of them: whole blocks, about as many each time, in a workspace for
    so many; the launches and the bits."""
    from tgo_b200.kernels.build import load_library
    o, N, P, T = ops(), 128, 64, 12000
    lib, a_head, chunks = load_library("state_space"), N * P + 3 * 64, T // 64 + 1
    lib.tgo_ssd_heads.restype = ctypes.c_int
    floats = chunks * (most * a_head + 4)
    plan = lib.tgo_ssd_heads(T, 1, H, G, N, P, ctypes.c_longlong(floats))
    assert plan % 65536 == at_once
    assert lib.tgo_ssd_heads(T, 1, H, G, N, P, ctypes.c_longlong(chunks * (at_once * a_head + 4))) == plan
    assert lib.tgo_ssd_heads(T, 1, H, G, N, P, ctypes.c_longlong(chunks * (a_head + 3))) == 0
    xbc, dt_raw = rnd(T, H * P + 2 * G * N, seed=N + P), rnd(T, H, seed=3).to(torch.bfloat16)
    a_log = torch.linspace(-3.0, 1.0, H, device=DEV)
    monkeypatch.setattr(o, "SSD_WORKSPACE_BYTES", 1 << 40)
    y, state = chunked_scan(o, monkeypatch, xbc, dt_raw, a_log, H, G, N, P)
    monkeypatch.setattr(o, "SSD_WORKSPACE_BYTES", 4 * floats)
    torch.cuda.synchronize()
    torch.cuda.reset_peak_memory_stats()
    launches, before = o.LAUNCHES[0], torch.cuda.memory_allocated()
    y2, state2 = chunked_scan(o, monkeypatch, xbc, dt_raw, a_log, H, G, N, P, chunks=None)
    taken = torch.cuda.max_memory_allocated() - before - 4 * (T * H * P + H * N * P)
    assert o.LAUNCHES[0] - launches == 4 * -(-H // at_once) and taken <= 4 * chunks * (at_once * a_head + 4) + 4096
    assert torch.equal(y, y2) and torch.equal(state, state2) and bool(y.any())


@pytest.mark.parametrize("H,G,N,P", [(4, 2, 128, 64), (2, 1, 64, 64), (3, 1, 128, 64), (3, 3, 64, 128), (2, 2, 128, 128)])
@pytest.mark.parametrize("lens", [[128], [1, 63, 64, 65, 200, 3], [700, 129]])
def test_selective_scan_by_chunks(H, G, N, P, lens, monkeypatch):
    """Requests that end before, on and after a chunk, fast and slow decays, against the recurrence
    in 64 bits: sums of at most N + 64 float32 terms behind at most eleven chunks."""
    o, T, B = ops(), sum(lens), len(lens)
    C = H * P + 2 * G * N
    xbc = rnd(T, C, seed=N + P)
    dt_raw = rnd(T, H + 2, seed=3).to(torch.bfloat16)[:, 1:H + 1]
    dt_bias, a_log, d = rnd(H, seed=4) - 2.0, torch.linspace(-3.0, 3.0, H, device=DEV), rnd(H, seed=5)
    floats = 8 + H * N * P + 12
    state = rnd(B + 2, floats, seed=6)
    before, slots = state.clone(), [5, 0, 3, 1, 7, 2][:B] if B > 2 else [2, 0][:B]
    starts = [0]
    for n in lens:
        starts.append(starts[-1] + n)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)       # noqa: E731
    y = torch.full((T, H * P), float("nan"), device=DEV)
    monkeypatch.setattr(o, "SSD_MIN_TOKENS", 1)
    launches = o.LAUNCHES[0]
    o.selective_scan(xbc, dt_raw, dt_bias, a_log, d, y, B, H, G, N, P, i32(starts), i32(slots), state, 8)
    assert o.LAUNCHES[0] == launches + 4                 # the chunked form ran
    x = xbc.double()
    u, bm, cm = x[:, :H * P].view(T, H, P), x[:, H * P:H * P + G * N].view(T, G, N), x[:, H * P + G * N:].view(T, G, N)
    bm, cm = (m.repeat_interleave(H // G, 1) for m in (bm, cm))
    dt = torch.nn.functional.softplus(dt_raw.double() + dt_bias.double())
    a = torch.exp(-torch.exp(a_log.double()) * dt)
    for b, n in enumerate(lens):
        S = before[slots[b], 8:8 + H * N * P].view(H, N, P).double()
        want = torch.empty(n, H, P, dtype=torch.float64, device=DEV)
        for i in range(n):
            t = starts[b] + i
            S = a[t][:, None, None] * S + bm[t][:, :, None] * (dt[t][:, None] * u[t])[:, None]
            want[i] = torch.einsum("hnp,hn->hp", S, cm[t]) + d.double()[:, None] * u[t]
        got = y[starts[b]:starts[b + 1]].view(n, H, P).double()
        assert (got - want).norm() <= 3e-6 * want.norm()
        assert (state[slots[b], 8:8 + H * N * P].view(H, N, P).double() - S).norm() <= 3e-6 * S.norm()
    after = state.clone()
    after[slots, 8:8 + H * N * P] = before[slots, 8:8 + H * N * P]
    assert torch.equal(after, before)


@pytest.mark.parametrize("n,groups", [(4, 3), (124, 2), (128, 16), (132, 1), (256, 5), (300, 2), (512, 8)])
@pytest.mark.parametrize("act,first", [(None, False), ("silu", True), ("sigmoid", False)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_gated_group_norm_in_fours(n, groups, act, first, dtype):
    """Groups read four channels at a time: whole and cut turns of 128, strided gates."""
    T, W = 37, n * groups
    o, gain = rnd(T, W, seed=n), rnd(W, seed=2)
    gate = rnd(T, W + 8, seed=3).to(dtype)[:, 4:W + 4] if act else None
    out = torch.empty(T, W, dtype=dtype, device=DEV)
    ops().gated_group_norm(o, gate, gain, out, groups, 1e-5, act, first)
    z = {None: 1.0, "silu": None, "sigmoid": None}[act]
    if act:
        z = gate.double() * torch.sigmoid(gate.double()) if act == "silu" else torch.sigmoid(gate.double())
    x = o.double() * (z if first else 1.0)
    want = (x.view(T, groups, n) * torch.rsqrt((x.view(T, groups, n) ** 2).mean(-1, keepdim=True) + 1e-5)).view(T, W)
    want = want * gain.double() * (1.0 if first else z)
    assert torch.allclose(out.double(), want, rtol=2.0 ** -8 if dtype == torch.bfloat16 else 1e-5, atol=1e-6)


@pytest.mark.parametrize("n,groups", [(516, 2), (1024, 1), (1028, 3), (1536, 1), (2048, 2)])
@pytest.mark.parametrize("act,first", [(None, False), ("silu", True)])
def test_gated_group_norm_a_block_a_group(n, groups, act, first):
    """Wider groups: four warps share one; cut turns of 512."""
    for dtype in (torch.float32, torch.bfloat16):
        test_gated_group_norm_in_fours(n, groups, act, first, dtype)


@pytest.mark.parametrize("n,groups", [(516, 2), (1024, 1), (1028, 3), (1536, 1), (2044, 2)])
@pytest.mark.parametrize("act,first", [(None, False), ("silu", True), ("sigmoid", False)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_gated_group_norm_the_same_bits_by_either_form(n, groups, act, first, dtype):
    """Gates and gains that begin off 16 bytes go a channel a lane: the same bits."""
    T, W, outs = 37, n * groups, []
    o, gain = rnd(T, W, seed=n), rnd(W, seed=2)
    gate = rnd(T, W, seed=3).to(dtype)
    for off in (0, 1):
        at = torch.empty(W + off, device=DEV)[off:]
        at.copy_(gain)
        outs.append(torch.empty(T, W, dtype=dtype, device=DEV))
        ops().gated_group_norm(o, gate if act else None, at, outs[-1], groups, 1e-5, act, first)
    assert torch.equal(*outs)


@pytest.mark.parametrize("H,dk,dv,ps", [(16, 576, 512, 16), (5, 576, 512, 8), (128, 264, 256, 64), (24, 200, 64, 32), (3, 448, 320, 128)])
@pytest.mark.parametrize("window,sink", [(0, False), (130, True), (300, False)])
def test_attention_latent_tc(H, dk, dv, ps, window, sink):
    """One wide row a token whose first channels are the values, on tcgen05: tiles of one to 42 tokens,
    one and two parts of the values, rows with a cut last block, pages inside and around a slot of 32
    keys, NaN in what nobody may read; against the generic kernel's float32 arithmetic. P and the
    result are rounded to bfloat16."""
    o, scale = ops(), dk ** -0.5
    assert o.attention_latent_tc_supports(H, dk, dv, ps)
    case = paged_case([150, 1, 40, 261], [333, 500, 0, 7], H, 1, dk, ps, torch.bfloat16, seed=dk + ps)
    if window:                                           # what lies before every window has gone back
        for b, f in enumerate(case["firsts"]):
            for i in range(max(0, f - window + 1) // ps):
                case["bt"][b, i] = 0
    sinks = rnd(H, seed=2) if sink else None
    t0, nt = attention_part().step_tiles(Ctx(case, False), 128 // H)
    T = case["q"].shape[0]
    out = torch.full((T, H * dv), 9.0, dtype=torch.bfloat16, device=DEV)
    o.attention_latent_tc(case["q"], out, H, dk, dv, case["kc"], ps, case["bt"], case["seq"], case["pos"], scale, window,
                          sinks, t0, nt)
    want = torch.empty(T, H * dv, device=DEV)
    kc = case["kc"].float()
    o.attention_generic(case["q"].float(), want, H, 1, dk, kc, kc, ps, case["bt"], case["seq"], case["pos"], scale, window,
                        value_dim=dv, sinks=sinks, value_row=dk)
    assert o.attention_latent_tc_error() == 0
    assert bool(torch.isfinite(want).all())
    assert torch.allclose(out.float(), want, **tol(torch.bfloat16))


def with_empty_requests(H, Hkv, dh, ps):
    """Prompt portions and single tokens in turn, every other single token one that brings nothing, more than
    a GPU's worth of items: blocks draw empty items between full ones, in both places of their rings."""
    extents = [40, 1, 1, 150, 1, 1, 1, 5] * 40
    firsts = [0, 30, 200, 60, 3, 500, 77, 9] * 40
    case = paged_case(extents, firsts, H, Hkv, dh, ps, torch.bfloat16, seed=dh)
    empty = torch.zeros(case["q"].shape[0], dtype=torch.bool, device=DEV)
    t = 0
    for i, n in enumerate(extents):
        if n == 1 and i % 2:
            empty[t] = True
        t += n
    case["pos"][empty] = -1
    return case, empty


@pytest.mark.parametrize("H,Hkv,dh,ps", [(4, 1, 64, 16), (8, 2, 128, 32)])
@pytest.mark.parametrize("extra", ["none", "sink", "all"])
def test_attention_tc_requests_that_bring_nothing(H, Hkv, dh, ps, extra):
    """Zeros for the tokens that bring nothing; the others as the generic kernel has them."""
    case, empty = with_empty_requests(H, Hkv, dh, ps)
    o, T, scale = ops(), case["q"].shape[0], dh ** -0.5
    kw = dict(softcap=2.0 if extra == "all" else 0.0, dist_bias=rnd(70, H, seed=1) if extra == "all" else None,
              sinks=rnd(H, seed=2) if extra != "none" else None,
              gate=rnd(T, H, seed=3).to(torch.bfloat16) if extra == "all" else None)
    t0, nt = attention_part().step_tiles(Ctx(case, False), 128 // (H // Hkv))
    out = torch.full_like(case["q"], 9.0)
    o.attention_tc_prefill(case["q"], out, H, Hkv, dh, case["kc"], case["vc"], ps, case["bt"], case["pos"],
                           case["seq"], t0, nt, scale, 100, own_counters=True, **kw)
    want = torch.empty_like(case["q"].float())
    kw["gate"] = kw["gate"].float() if kw["gate"] is not None else None
    o.attention_generic(case["q"].float(), want, H, Hkv, dh, case["kc"].float(), case["vc"].float(), ps, case["bt"],
                        case["seq"], case["pos"], scale, 100, **kw)
    assert o.attention_tc_error() == 0 and bool(torch.isfinite(want).all())
    assert not out[empty].any() and torch.allclose(out.float(), want, **tol(torch.bfloat16))


@pytest.mark.parametrize("H,dk,dv,ps", [(16, 576, 512, 16), (40, 200, 64, 32)])
@pytest.mark.parametrize("sink", [False, True])
def test_attention_latent_tc_requests_that_bring_nothing(H, dk, dv, ps, sink):
    """Zeros for the tokens that bring nothing; the others as the generic kernel has them."""
    case, empty = with_empty_requests(H, 1, dk, ps)
    o, T, scale = ops(), case["q"].shape[0], dk ** -0.5
    sinks = rnd(H, seed=2) if sink else None
    t0, nt = attention_part().step_tiles(Ctx(case, False), 128 // H)
    out = torch.full((T, H * dv), 9.0, dtype=torch.bfloat16, device=DEV)
    o.attention_latent_tc(case["q"], out, H, dk, dv, case["kc"], ps, case["bt"], case["seq"], case["pos"], scale, 0,
                          sinks, t0, nt)
    want, kc = torch.empty(T, H * dv, device=DEV), case["kc"].float()
    o.attention_generic(case["q"].float(), want, H, 1, dk, kc, kc, ps, case["bt"], case["seq"], case["pos"], scale, 0,
                        value_dim=dv, sinks=sinks, value_row=dk)
    assert o.attention_latent_tc_error() == 0 and bool(torch.isfinite(want).all())
    assert not out[empty].any() and torch.allclose(out.float(), want, **tol(torch.bfloat16))


@pytest.mark.parametrize("H,Hkv,ps", [(16, 4, 16), (5, 1, 8), (12, 1, 32), (16, 2, 64)])
@pytest.mark.parametrize("window,keep", [(0, 0), (130, 0), (140, 5), (300, 200)])
@pytest.mark.parametrize("extra", ["sink", "cap", "bias", "all"])
def test_attention_sink_decode_tma(H, Hkv, ps, window, keep, extra):
    """Single tokens with a sink, kept first keys, bounded scores, a bias by distance and a gate, keys
    whole and cut in shares (some empty), against the generic kernel's float32 arithmetic."""
    dh, o = 128, ops()
    case = paged_case([1, 1, 1, 1, 1], [0, 63, 64, 700, 333], H, Hkv, dh, ps, torch.bfloat16, seed=ps)
    case["pos"][0] = -1                                   # a request that brings nothing
    T = case["q"].shape[0]
    if keep:                                              # what lies between has gone back
        for b, f in enumerate(case["firsts"]):
            for i in range(-(-keep // ps), max(0, f - window + 1) // ps):
                case["bt"][b, i] = 0
    kw = dict(softcap=2.0 if extra in ("cap", "all") else 0.0, keep_first=keep,
              dist_bias=rnd(70, H, seed=1) if extra in ("bias", "all") else None,
              gate=rnd(T, H, seed=3).to(torch.bfloat16) if extra == "all" else None)
    sinks = rnd(H, seed=2) if extra in ("sink", "all") else None
    want = torch.empty_like(case["q"].float())
    kw32 = dict(kw, gate=kw["gate"].float() if kw["gate"] is not None else None)
    o.attention_generic(case["q"].float(), want, H, Hkv, dh, case["kc"].float(), case["vc"].float(), ps, case["bt"],
                        case["seq"], case["pos"], dh ** -0.5, window, sinks=sinks, **kw32)
    assert bool(torch.isfinite(want).all())
    for splits in (1, 3, 16):
        out = torch.full_like(case["q"], 9.0)
        o.attention_sink_decode_tma(case["q"], out, H, Hkv, dh, case["kc"], case["vc"], ps, case["bt"], case["seq"],
                                    case["pos"], dh ** -0.5, window, sinks, splits, **kw)
        assert o.attention_decode_tma_error() == 0
        assert torch.allclose(out.float(), want, **tol(torch.bfloat16)), splits
