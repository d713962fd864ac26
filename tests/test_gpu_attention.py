"""Causal GQA attention forward/backward on the GPU against the oracle: the
reference layout ops (FLASH / ROWDOT / FLASH_BWD on [B,H,T,DH], fp32 outputs)
and the fused ops on [B,T,H,DH]; fp32 and bf16; head_dim 16..128; ragged T;
MHA / GQA / MQA; determinism."""
import ctypes

import numpy as np
import pytest

from axis_b200 import engine as E
from axis_b200.engine import Engine, op
from oracle import step_numpy as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def eng():
    e = Engine()
    e.alloc(4)
    yield e
    e.shutdown()


def bf(a):
    return E.bf16_bits_to_f32(E.f32_to_bf16_bits(a))


def put(eng, arr, dt):
    i = eng.alloc(arr.size, 2 if dt else 4)
    eng.upload_bf16(i, arr) if dt else eng.upload(i, arr)
    return i


def get(eng, i, shape, dt):
    return eng.download_bf16(i, shape) if dt else eng.download(i, shape)


def rel(got, ref):
    return float(np.abs(got - ref).max() / (np.abs(ref).max() + 1e-9))


def make(rng, B, H, KV, T, DH, dt):
    q = rng.standard_normal((B, H, T, DH)).astype(np.float32)
    k = rng.standard_normal((B, KV, T, DH)).astype(np.float32)
    v = rng.standard_normal((B, KV, T, DH)).astype(np.float32)
    do = rng.standard_normal((B, H, T, DH)).astype(np.float32)
    if dt:
        q, k, v, do = bf(q), bf(k), bf(v), bf(do)
    return q, k, v, do


CASES = [(2, 4, 2, 32, 32), (1, 6, 2, 17, 16), (2, 2, 2, 64, 64), (1, 4, 1, 40, 128), (1, 3, 3, 130, 64),
         # head_dim 64 with whole 128-token tiles: the tcgen05 kernels when fallback == 0
         (1, 4, 4, 128, 64), (2, 6, 2, 256, 64), (2, 3, 1, 384, 64), (1, 4, 2, 1024, 64),
         # head_dim 128 with whole tiles: the head_dim-128 tcgen05 kernels when fallback == 0
         (1, 2, 2, 128, 128), (2, 4, 2, 256, 128), (1, 3, 1, 640, 128)]


@pytest.mark.parametrize("dt", [0, 1])
@pytest.mark.parametrize("B,H,KV,T,DH", CASES)
@pytest.mark.parametrize("fallback", [0, 2])
def test_fused_attention_bthd(eng, dt, B, H, KV, T, DH, fallback):
    rng = np.random.default_rng(T * DH + H)
    q, k, v, do = make(rng, B, H, KV, T, DH, dt)
    scale = 1.0 / np.sqrt(DH)
    o_ref, lse_ref = O.attention_fwd(q, k, v, scale)
    t = lambda x: np.ascontiguousarray(x.transpose(0, 2, 1, 3))
    iq, ik, iv, ido = put(eng, t(q), dt), put(eng, t(k), dt), put(eng, t(v), dt), put(eng, t(do), dt)
    # scratch of the backward: D = rowsum(dO*O) followed by the fp32 dQ accumulator of the tensor-core path
    io, ilse, iD = eng.alloc(q.size), eng.alloc(B * H * T), eng.alloc(B * H * T + q.size)
    idq, idk, idv = eng.alloc(q.size), eng.alloc(k.size), eng.alloc(k.size)
    eng.set_fallback(fallback)
    eng.run([op(E.ATTN_FWD, a=iq, b=ik, d=iv, c=io, sa=ilse, m=T, n=DH, k=KV, batch=B, tb=H, dt=dt, alpha=scale)])
    o = get(eng, io, (B, T, H, DH), dt).transpose(0, 2, 1, 3)
    lse = eng.download(ilse, (B, H, T))
    lim = 1.5e-2 if dt else 2e-5
    assert rel(o, o_ref) <= lim
    assert np.abs(lse - lse_ref).max() <= (2e-2 if dt else 2e-5)
    o_in = bf(o) if dt else o
    dq_ref, dk_ref, dv_ref = O.attention_bwd(q, k, v, do, scale)
    eng.launch_count(reset=True)
    eng.run([op(E.ATTN_BWD, a=iq, b=ik, d=iv, c=ido, sa=ilse, sb=io, tb=idq, sc=idk, oa=idv, ob=H, oc=iD,
                m=T, n=DH, k=KV, batch=B, dt=dt, alpha=scale)])
    eng.set_fallback(0)
    # row dots, main kernel and conversion of dQ on tcgen05; row dots, dQ and dK / dV elsewhere
    assert eng.launch_count() == 3
    dq = get(eng, idq, (B, T, H, DH), dt).transpose(0, 2, 1, 3)
    dk = get(eng, idk, (B, T, KV, DH), dt).transpose(0, 2, 1, 3)
    dv = get(eng, idv, (B, T, KV, DH), dt).transpose(0, 2, 1, 3)
    lim = 2e-2 if dt else 3e-5
    assert rel(dq, dq_ref) <= lim and rel(dk, dk_ref) <= lim and rel(dv, dv_ref) <= lim
    assert eng.device_status() == 0


def test_reference_layout_flash_ops(eng):
    """FLASH -> (permute) -> ROWDOT on [B,T,H,DH] -> FLASH_BWD into fp32 buffers, as the
    reference plan chains them (axis/compile.py:329-331, 406-421)."""
    rng = np.random.default_rng(0)
    B, H, KV, T, DH = 2, 4, 2, 48, 32
    q, k, v, do = make(rng, B, H, KV, T, DH, 1)
    scale = 1.0 / np.sqrt(DH)
    iq, ik, iv, ido = put(eng, q, 1), put(eng, k, 1), put(eng, v, 1), put(eng, do, 1)
    io, ilse = eng.alloc(q.size, 2), eng.alloc(B * H * T)
    eng.run([op(E.FLASH, a=iq, b=ik, d=iv, c=io, m=T, n=DH, k=KV, batch=B, tb=H, sa=ilse, dt=1, alpha=scale)])
    o_ref, lse_ref = O.attention_fwd(q, k, v, scale)
    o = eng.download_bf16(io, q.shape)
    assert rel(o, o_ref) <= 1.5e-2
    assert np.abs(eng.download(ilse, (B, H, T)) - lse_ref).max() <= 2e-2
    io2, ido2, iD = eng.alloc(q.size, 2), eng.alloc(q.size, 2), eng.alloc(B * T * H)
    idq, idk, idv = eng.alloc(q.size), eng.alloc(k.size), eng.alloc(k.size)
    eng.run([op(E.PERM_0213, a=io, c=io2, m=B, n=H, k=T, batch=DH, dt=1),
             op(E.PERM_0213, a=ido, c=ido2, m=B, n=H, k=T, batch=DH, dt=1),
             op(E.ROWDOT, a=ido2, b=io2, c=iD, m=B * T * H, n=DH, dt=1),
             op(E.SCALE, a=idq, c=idq, n=q.size, alpha=0.0), op(E.SCALE, a=idk, c=idk, n=k.size, alpha=0.0),
             op(E.SCALE, a=idv, c=idv, n=k.size, alpha=0.0),
             op(E.FLASH_BWD, a=iq, b=ik, d=iv, c=ido, sa=ilse, sb=iD, tb=idq, sc=idk, oa=idv, ob=H,
                m=T, n=DH, k=KV, batch=B, dt=1, alpha=scale)])
    dq_ref, dk_ref, dv_ref = O.attention_bwd(q, k, v, do, scale)
    assert rel(eng.download(idq, q.shape), dq_ref) <= 2e-2
    assert rel(eng.download(idk, k.shape), dk_ref) <= 2e-2
    assert rel(eng.download(idv, k.shape), dv_ref) <= 2e-2


@pytest.mark.parametrize("T", [256, 1024])
@pytest.mark.parametrize("DH", [64, 128])
@pytest.mark.parametrize("fallback", [0, 2])
def test_attention_backward_is_deterministic(eng, fallback, DH, T):
    """dK/dV are summed on chip in a fixed order in both paths.  dQ is bit-stable in the
    general path; the tensor-core path adds its per-key-tile dQ pieces with an unordered
    fp32 reduce-add (as the reference's atomics do), so dQ is only checked there for
    closeness."""
    rng = np.random.default_rng(1)
    B, H, KV = 1, 6, 2         # T = 1024: eight key tiles, deep pipelines (ring slots and TMEM buffers reused many times)
    q, k, v, do = make(rng, B, H, KV, T, DH, 1)
    t = lambda x: np.ascontiguousarray(x.transpose(0, 2, 1, 3))
    iq, ik, iv, ido = put(eng, t(q), 1), put(eng, t(k), 1), put(eng, t(v), 1), put(eng, t(do), 1)
    io, ilse, iD = eng.alloc(q.size, 2), eng.alloc(B * H * T), eng.alloc(B * H * T + q.size)
    idq, idk, idv = eng.alloc(q.size, 2), eng.alloc(k.size, 2), eng.alloc(k.size, 2)
    plan = [op(E.ATTN_FWD, a=iq, b=ik, d=iv, c=io, sa=ilse, m=T, n=DH, k=KV, batch=B, tb=H, dt=1, alpha=0.125),
            op(E.ATTN_BWD, a=iq, b=ik, d=iv, c=ido, sa=ilse, sb=io, tb=idq, sc=idk, oa=idv, ob=H, oc=iD,
               m=T, n=DH, k=KV, batch=B, dt=1, alpha=0.125)]
    eng.set_fallback(fallback)
    eng.run(plan)
    first = [eng.download_raw(i, n, np.uint16) for i, n in ((idq, q.size), (idk, k.size), (idv, k.size))]
    for _ in range(3):
        eng.run(plan)
        for which, (f, (i, n)) in enumerate(zip(first, ((idq, q.size), (idk, k.size), (idv, k.size)))):
            again = eng.download_raw(i, n, np.uint16)
            if which == 0 and fallback == 0:
                a, b2 = E.bf16_bits_to_f32(f), E.bf16_bits_to_f32(again)
                assert np.abs(a - b2).max() <= 1e-2 * np.abs(a).max()
            else:
                assert np.array_equal(f, again)
    eng.set_fallback(0)
    assert eng.device_status() == 0


@pytest.mark.parametrize("dt,B,H,KV,T,DH", [(1, 2, 6, 2, 256, 64), (1, 1, 4, 2, 256, 128), (0, 1, 4, 2, 40, 32), (1, 1, 3, 1, 130, 64)])
def test_attention_backward_with_the_inverse_rotary_inside(eng, dt, B, H, KV, T, DH):
    """ATTN_BWD with gamma > 0 returns dq and dk already rotated back (the compiled step's form): the head_dim-64
    tensor-core kernel applies the rotation before rounding, every other path runs the rotary kernel behind the
    attention kernels.  Reference: attention_bwd followed by rope_bwd of the oracle."""
    rng = np.random.default_rng(7 * T + DH)
    q, k, v, do = make(rng, B, H, KV, T, DH, dt)
    scale = 1.0 / np.sqrt(DH)
    cos, sin = O.rope_tables(T, DH)
    t = lambda x: np.ascontiguousarray(x.transpose(0, 2, 1, 3))
    iq, ik, iv, ido = put(eng, t(q), dt), put(eng, t(k), dt), put(eng, t(v), dt), put(eng, t(do), dt)
    ic, isn = put(eng, cos, 0), put(eng, sin, 0)
    io, ilse, iD = eng.alloc(q.size), eng.alloc(B * H * T), eng.alloc(B * H * T + q.size)
    idq, idk, idv = eng.alloc(q.size), eng.alloc(k.size), eng.alloc(k.size)
    eng.run([op(E.ATTN_FWD, a=iq, b=ik, d=iv, c=io, sa=ilse, m=T, n=DH, k=KV, batch=B, tb=H, dt=dt, alpha=scale),
             op(E.ATTN_BWD, a=iq, b=ik, d=iv, c=ido, sa=ilse, sb=io, tb=idq, sc=idk, oa=idv, ob=H, oc=iD,
                m=T, n=DH, k=KV, batch=B, dt=dt, alpha=scale, beta=float(ic), gamma=float(isn))])
    dq_ref, dk_ref, dv_ref = O.attention_bwd(q, k, v, do, scale)
    dq_ref, dk_ref = O.rope_bwd(dq_ref, cos, sin), O.rope_bwd(dk_ref, cos, sin)
    dq = get(eng, idq, (B, T, H, DH), dt).transpose(0, 2, 1, 3)
    dk = get(eng, idk, (B, T, KV, DH), dt).transpose(0, 2, 1, 3)
    dv = get(eng, idv, (B, T, KV, DH), dt).transpose(0, 2, 1, 3)
    lim = 2e-2 if dt else 3e-5
    assert rel(dq, dq_ref) <= lim and rel(dk, dk_ref) <= lim and rel(dv, dv_ref) <= lim
    assert eng.device_status() == 0


@pytest.mark.parametrize("B,H,KV,T,DH", [
    (1, 2, 1, 1, 64), (2, 3, 3, 63, 64), (1, 4, 2, 127, 64), (2, 2, 1, 129, 64), (1, 6, 2, 321, 64), (2, 4, 2, 1000, 64),
    (1, 2, 2, 128, 8), (2, 8, 4, 256, 32), (1, 3, 1, 130, 40),
    (1, 2, 1, 65, 72), (2, 2, 2, 200, 96), (1, 4, 2, 385, 128), (1, 2, 1, 1, 128)])
def test_attention_on_ragged_tiles_and_narrow_heads(eng, B, H, KV, T, DH):
    """Sequences that end inside a tile and heads narrower than the columns of a tile (`attn_mma.cu`; T 1000 `attn_tcs.cu`), with guard rows behind every
    output (a store past the end of the sequence or the head would land there).  Tolerances: operands and results are bf16
    (half an ulp, 2^-8 at most) with fp32 sums over up to 1000 keys or queries, the largest element of a result is the scale: the limits of
    the whole-tile cases above are more than enough."""
    rng = np.random.default_rng(T * DH + H)
    q, k, v, do = make(rng, B, H, KV, T, DH, 1)
    scale = 1.0 / np.sqrt(DH)
    t = lambda x: np.ascontiguousarray(x.transpose(0, 2, 1, 3))
    iq, ik, iv, ido = put(eng, t(q), 1), put(eng, t(k), 1), put(eng, t(v), 1), put(eng, t(do), 1)
    Tp = (T + 127) // 128 * 128
    guard = 4096
    outs = {n: eng.alloc(a.size + guard, 2) for n, a in (("o", q), ("dq", q), ("dk", k), ("dv", k))}
    mark = np.full(q.size + guard, 0x7fc1, dtype=np.uint16)
    for n, i in outs.items():
        eng.upload_raw(i, mark[:(q if n in ("o", "dq") else k).size + guard])
    ilse, iD = eng.alloc(B * H * T), eng.alloc(2 * B * H * Tp + q.size)
    eng.run([op(E.ATTN_FWD, a=iq, b=ik, d=iv, c=outs["o"], sa=ilse, m=T, n=DH, k=KV, batch=B, tb=H, dt=1, alpha=scale)])
    eng.launch_count(reset=True)
    eng.run([op(E.ATTN_BWD, a=iq, b=ik, d=iv, c=ido, sa=ilse, sb=outs["o"], tb=outs["dq"], sc=outs["dk"], oa=outs["dv"], ob=H,
                oc=iD, m=T, n=DH, k=KV, batch=B, dt=1, alpha=scale)])
    assert eng.launch_count() == 3                          # row dots, dQ, dK / dV
    assert eng.device_status() == 0
    o_ref, lse_ref = O.attention_fwd(q, k, v, scale)
    ref = dict(zip(("dq", "dk", "dv"), O.attention_bwd(q, k, v, do, scale)), o=o_ref)
    assert np.abs(eng.download(ilse, (B, H, T)) - lse_ref).max() <= 2e-2
    for n, i in outs.items():
        heads = H if n in ("o", "dq") else KV
        raw = eng.download_raw(i, B * T * heads * DH + guard, np.uint16)
        assert np.all(raw[-guard:] == 0x7fc1), n
        got = E.bf16_bits_to_f32(raw[:-guard]).reshape(B, T, heads, DH).transpose(0, 2, 1, 3)
        assert np.isfinite(got).all(), n
        if T == 1 and n in ("dq", "dk"):                    # a single key: P = 1 and dS = dP - D is rounding alone
            assert np.abs(got).max() <= 2e-2 * np.abs(do).max() * np.abs(v).max() * DH * scale
        else:
            assert rel(got, ref[n]) <= (1.5e-2 if n == "o" else 2e-2), n


def attention_f64(q, k, v, do, scale):
    """o, dq, dk, dv in float64"""
    q, k, v, do = (x.astype(np.float64) for x in (q, k, v, do))
    B, H, T, DH = q.shape
    KV = k.shape[1]
    kk, vv = np.repeat(k, H // KV, axis=1), np.repeat(v, H // KV, axis=1)
    s = np.where(np.tril(np.ones((T, T), dtype=bool)), scale * (q @ kk.transpose(0, 1, 3, 2)), -np.inf)
    p = np.exp(s - s.max(-1, keepdims=True))
    p /= p.sum(-1, keepdims=True)
    o = p @ vv
    ds = p * (do @ vv.transpose(0, 1, 3, 2) - (do * o).sum(-1, keepdims=True)) * scale
    group = lambda x: x.reshape(B, KV, H // KV, T, DH).sum(2)
    return dict(o=o, dq=ds @ kk, dk=group(ds.transpose(0, 1, 3, 2) @ q), dv=group(p.transpose(0, 1, 3, 2) @ do))


def run_bf16_attention(eng, q, k, v, do, scale, fallback, times=1, rotary=()):
    """o, dq, dk, dv as bf16 bits in [B,T,heads,DH], one list per run; rotary: cos and sin tables for dq and dk to be rotated back"""
    B, H, T, DH = q.shape
    KV = k.shape[1]
    t = lambda x: np.ascontiguousarray(x.transpose(0, 2, 1, 3))
    iq, ik, iv, ido = put(eng, t(q), 1), put(eng, t(k), 1), put(eng, t(v), 1), put(eng, t(do), 1)
    out = {n: (eng.alloc(a.size, 2), (B, T, a.shape[1], DH)) for n, a in (("o", q), ("dq", q), ("dk", k), ("dv", k))}
    ilse, iD = eng.alloc(B * H * T), eng.alloc(2 * B * H * (T + 128) + q.size)
    tables = dict(zip(("beta", "gamma"), (float(put(eng, x, 0)) for x in rotary)))
    eng.set_fallback(fallback)
    runs = []
    for _ in range(times):
        eng.run([op(E.ATTN_FWD, a=iq, b=ik, d=iv, c=out["o"][0], sa=ilse, m=T, n=DH, k=KV, batch=B, tb=H, dt=1, alpha=scale),
                 op(E.ATTN_BWD, a=iq, b=ik, d=iv, c=ido, sa=ilse, sb=out["o"][0], tb=out["dq"][0], sc=out["dk"][0], oa=out["dv"][0],
                    ob=H, oc=iD, m=T, n=DH, k=KV, batch=B, dt=1, alpha=scale, **tables)])
        runs.append({n: eng.download_raw(i, sh, np.uint16) for n, (i, sh) in out.items()})
    eng.set_fallback(0)
    assert eng.device_status() == 0
    return runs


@pytest.mark.parametrize("B,H,KV,T,DH", [(1, 4, 2, 1000, 64), (1, 6, 2, 321, 64), (2, 8, 4, 256, 32), (1, 3, 1, 130, 40),
                                         (2, 2, 2, 200, 96), (1, 4, 2, 385, 128),
                                         (8, 24, 8, 320, 64), (16, 16, 16, 130, 64)])       # on tcgen05; the backward without clusters
def test_attention_of_other_shapes_keeps_fp32_probabilities(eng, B, H, KV, T, DH):
    """Shapes that the whole-tile tcgen05 kernels do not take had P and dS in fp32 on the general kernels (fallback 2) and the same bits on
    every run; the tensor-core kernels for them (attn_mma.cu, and attn_tcs.cu for (8, 24, 8, 320, 64) and T 1000) may be no further from float64 than those and as reproducible.  P and dS enter
    as two bf16 numbers, off by at most 2^-17 of an element; the results' own rounding to bf16 is up to 2^-8, so the 2-norm error
    grows by a part in 2^18, and the bound of one per cent leaves room for results that round the other way."""
    rng = np.random.default_rng(T + DH)
    q, k, v, do = make(rng, B, H, KV, T, DH, 1)
    scale = 1.0 / np.sqrt(DH)
    ref = attention_f64(q, k, v, do, scale)
    runs = run_bf16_attention(eng, q, k, v, do, scale, 0, times=4)
    general = run_bf16_attention(eng, q, k, v, do, scale, 2)[0]
    for n, exact in ref.items():
        assert all(np.array_equal(runs[0][n], r[n]) for r in runs[1:]), n
        err = lambda bits: float(np.linalg.norm(E.bf16_bits_to_f32(bits).transpose(0, 2, 1, 3) - exact) / np.linalg.norm(exact))
        assert err(runs[0][n]) <= 1.01 * err(general[n]), (n, err(runs[0][n]), err(general[n]))


@pytest.mark.parametrize("B,H,KV,T,DH", [(2, 8, 4, 256, 32), (1, 2, 1, 225, 8), (1, 4, 2, 97, 40), (1, 3, 3, 130, 128), (1, 2, 1, 64, 256), (16, 8, 8, 65, 64),
                                             (1, 4, 1, 33, 1), (2, 2, 2, 40, 2), (1, 8, 4, 150, 4), (1, 8, 1, 96, 256)])
def test_fp32_attention_over_clusters(eng, B, H, KV, T, DH):
    """Few rows: clusters of two to eight CTAs share a block's tiles, some of them without one ((16, 8, 8, 65, 64) fills the SMs).  Head dims of 32, 40 and 64 run on attn_f32.cu
    here, on the general kernels in the test below.  Sums of T products of N(0,1) numbers in fp32 in any order err by less than 2^-24 sqrt(T) a term: 2e-5 of the largest
    result, as for one CTA; a second run gives the same bits."""
    rng = np.random.default_rng(T + DH)
    q, k, v, do = make(rng, B, H, KV, T, DH, 0)
    scale = 1.0 / np.sqrt(DH)
    t = lambda x: np.ascontiguousarray(x.transpose(0, 2, 1, 3))
    iq, ik, iv, ido = put(eng, t(q), 0), put(eng, t(k), 0), put(eng, t(v), 0), put(eng, t(do), 0)
    out = {n: (eng.alloc(a.size), a.shape[1]) for n, a in (("o", q), ("dq", q), ("dk", k), ("dv", k))}
    ilse, iD = eng.alloc(B * H * T), eng.alloc(B * H * T)
    runs = []
    for _ in range(2):
        eng.run([op(E.ATTN_FWD, a=iq, b=ik, d=iv, c=out["o"][0], sa=ilse, m=T, n=DH, k=KV, batch=B, tb=H, dt=0, alpha=scale),
                 op(E.ATTN_BWD, a=iq, b=ik, d=iv, c=ido, sa=ilse, sb=out["o"][0], tb=out["dq"][0], sc=out["dk"][0], oa=out["dv"][0],
                    ob=H, oc=iD, m=T, n=DH, k=KV, batch=B, dt=0, alpha=scale)])
        runs.append({n: eng.download(i, (B, T, heads, DH)).transpose(0, 2, 1, 3) for n, (i, heads) in out.items()})
    lse = eng.download(ilse, (B, H, T))
    for n, ref in attention_f64(q, k, v, do, scale).items():
        assert np.array_equal(runs[0][n], runs[1][n]), n
        assert np.abs(runs[0][n] - ref).max() <= 2e-5 * np.abs(ref).max(), n
    assert np.abs(lse - O.attention_fwd(q, k, v, scale)[1]).max() <= 2e-5
    assert eng.device_status() == 0


@pytest.mark.parametrize("B,H,KV,T,DH,off", [
    (2, 8, 4, 256, 32, 1), (1, 4, 2, 97, 40, 1), (16, 8, 8, 65, 64, 1), (1, 4, 1, 300, 64, 1), (3, 6, 2, 70, 12, 1),       # head dims of attn_f32.cu from buffers that it does not take
    (1, 4, 2, 150, 63, 0), (24, 8, 8, 65, 50, 0), (2, 8, 4, 120, 34, 0), (20, 16, 16, 64, 72, 0)])                         # head dims of none of it
def test_fp32_attention_on_the_general_kernels(eng, B, H, KV, T, DH, off):
    """Shared walks and blocks of their own ((16, 8, 8, 65, 64), (24, 8, 8, 65, 50) and the last fill the SMs) by the variant that ran, bounds as in the test above."""
    rng = np.random.default_rng(T + DH)
    q, k, v, do = make(rng, B, H, KV, T, DH, 0)
    scale = 1.0 / np.sqrt(DH)

    def placed(size, arr=None):                          # a buffer that starts `off` floats into its allocation
        i = eng.view(eng.alloc(size + off), 4 * off, 4 * size)
        if arr is not None:
            eng.upload(i, np.ascontiguousarray(arr.transpose(0, 2, 1, 3)))
        return i
    iq, ik, iv, ido = (placed(x.size, x) for x in (q, k, v, do))
    out = {n: (placed(a.size), a.shape[1]) for n, a in (("o", q), ("dq", q), ("dk", k), ("dv", k))}
    ilse, iD = eng.alloc(B * H * T), eng.alloc(B * H * T)
    runs = []
    for _ in range(2):
        eng.run([op(E.ATTN_FWD, a=iq, b=ik, d=iv, c=out["o"][0], sa=ilse, m=T, n=DH, k=KV, batch=B, tb=H, dt=0, alpha=scale)])
        assert eng.last_variant() == 0x86
        eng.run([op(E.ATTN_BWD, a=iq, b=ik, d=iv, c=ido, sa=ilse, sb=out["o"][0], tb=out["dq"][0], sc=out["dk"][0], oa=out["dv"][0], ob=H, oc=iD, m=T, n=DH, k=KV,
                    batch=B, dt=0, alpha=scale)])
        assert eng.last_variant() == 0x87
        runs.append({n: eng.download(i, (B, T, heads, DH)).transpose(0, 2, 1, 3) for n, (i, heads) in out.items()})
    for n, ref in attention_f64(q, k, v, do, scale).items():
        assert np.array_equal(runs[0][n], runs[1][n]), n
        assert np.abs(runs[0][n] - ref).max() <= 2e-5 * np.abs(ref).max(), n
    assert np.abs(eng.download(ilse, (B, H, T)) - O.attention_fwd(q, k, v, scale)[1]).max() <= 2e-5
    assert eng.device_status() == 0


@pytest.mark.parametrize("B,H,KV,T,DH", [(3, 8, 8, 26, 12), (4, 1, 1, 27, 64), (2, 12, 12, 71, 12), (6, 3, 1, 12, 40)])
def test_short_fp32_attention_takes_no_longer_than_on_the_general_kernels(eng, B, H, KV, T, DH):
    """Backward from aligned buffers against the general kernels (from buffers that start one float later).  us on one B200, aligned and there / here whatever the shape / now: 8.9 / 20.2 / 8.9,
    13.7 / 29.4 / 13.7, 17.7 / 25.6 / 17.5, 18.4 / 25.6 / 14.7."""
    rng = np.random.default_rng(T)
    q, k, v, do = make(rng, B, H, KV, T, DH, 0)
    times = []
    for off in (0, 1):
        placed = lambda x: eng.view(eng.alloc(x.size + off), 4 * off, 4 * x.size)
        ins = [placed(x) for x in (q, k, v, do)]
        for i, x in zip(ins, (q, k, v, do)):
            eng.upload(i, np.ascontiguousarray(x.transpose(0, 2, 1, 3)))
        io, idq, idk, idv, ilse, iD = placed(q), placed(q), placed(k), placed(k), eng.alloc(B * H * T), eng.alloc(B * H * T)
        eng.run([op(E.ATTN_FWD, a=ins[0], b=ins[1], d=ins[2], c=io, sa=ilse, m=T, n=DH, k=KV, batch=B, tb=H, dt=0, alpha=DH ** -0.5)])
        plan = [op(E.ATTN_BWD, a=ins[0], b=ins[1], d=ins[2], c=ins[3], sa=ilse, sb=io, tb=idq, sc=idk, oa=idv, ob=H, oc=iD, m=T, n=DH, k=KV, batch=B, dt=0, alpha=DH ** -0.5)] * 20
        eng.capture(plan)
        ms = ctypes.c_float(0)
        runs = []
        for _ in range(6):
            assert eng.lib.eng_time_replay(5, ctypes.byref(ms)) == 0
            runs.append(ms.value)
        times.append(min(runs))
    assert times[0] <= 1.1 * times[1], times


@pytest.mark.parametrize("B,H,KV,T,DH,gain", [
    (40, 8, 4, 3, 64, 1), (20, 16, 8, 64, 48, 1), (20, 16, 8, 65, 64, 1),       # one tile: a piece of a step, one step, two
    (4, 12, 4, 129, 64, 1), (2, 16, 2, 500, 56, 1),                             # dK / dV over clusters of two and four, some CTAs with no step
    (1, 10, 5, 1000, 64, 6), (1, 8, 8, 1300, 40, 1)])                           # scores that move the running maximum; a narrow head
def test_attention_with_split_probabilities_on_tcgen05(eng, B, H, KV, T, DH, gain):
    """The shapes of the test above that fill the GPU, on the tcgen05 kernels, with the same bound against float64 and on every run;
    gain spreads the scores, so that rows of the forward rescale."""
    rng = np.random.default_rng(T + DH)
    q, k, v, do = make(rng, B, H, KV, T, DH, 1)
    scale = gain / np.sqrt(DH)
    runs = run_bf16_attention(eng, q, k, v, do, scale, 0, times=3)
    assert eng.last_variant() == 0x81
    general = run_bf16_attention(eng, q, k, v, do, scale, 2)[0]
    for n, exact in attention_f64(q, k, v, do, scale).items():
        assert all(np.array_equal(runs[0][n], r[n]) for r in runs[1:]), n
        err = lambda bits: float(np.linalg.norm(E.bf16_bits_to_f32(bits).transpose(0, 2, 1, 3) - exact) / np.linalg.norm(exact))
        assert err(runs[0][n]) <= 1.01 * err(general[n]), (n, err(runs[0][n]), err(general[n]))


@pytest.mark.parametrize("B,H,KV,T,DH,parts,launches", [
    (4, 24, 8, 500, 64, 1, 3), (4, 12, 4, 129, 64, 2, 3), (2, 16, 2, 900, 64, 4, 3),       # rotated before they are rounded
    (2, 16, 8, 500, 48, 2, 4), (4, 16, 16, 130, 40, 1, 4)])                                # the rotary as a launch of its own
def test_split_probabilities_on_tcgen05_with_the_inverse_rotary_inside(eng, B, H, KV, T, DH, parts, launches):
    """dq and dk of the tcgen05 backward leave ATTN_BWD rotated back, from one CTA to a key tile and from clusters: no further from float64 than the
    general kernels, which round to bf16 in front of the rotation and behind it, and within that much (a wrong row, sign or pair of the
    tables errs by as much as the result).  dv is not rotated."""
    assert eng.lib.eng_attn_route(1, B, H, KV, T, DH) == parts
    rng = np.random.default_rng(T + DH)
    q, k, v, do = make(rng, B, H, KV, T, DH, 1)
    scale = 1.0 / np.sqrt(DH)
    cos, sin = O.rope_tables(T, DH)
    eng.launch_count(reset=True)
    runs = run_bf16_attention(eng, q, k, v, do, scale, 0, times=2, rotary=(cos, sin))
    assert eng.last_variant() == 0x81 and eng.launch_count() == 2 * (1 + launches)
    general = run_bf16_attention(eng, q, k, v, do, scale, 2, rotary=(cos, sin))[0]
    ref = attention_f64(q, k, v, do, scale)
    c, s = cos.astype(np.float64), sin.astype(np.float64)
    for n in ("dq", "dk"):
        g1, g2 = ref[n][..., :DH // 2], ref[n][..., DH // 2:]
        ref[n] = np.concatenate([g1 * c + g2 * s, g2 * c - g1 * s], -1)
    for n, exact in ref.items():
        assert np.array_equal(runs[0][n], runs[1][n]), n
        err = lambda bits: float(np.linalg.norm(E.bf16_bits_to_f32(bits).transpose(0, 2, 1, 3) - exact) / np.linalg.norm(exact))
        assert err(runs[0][n]) <= 1.01 * err(general[n]) <= 1.01 * 2.0 ** -7, (n, err(runs[0][n]), err(general[n]))


@pytest.mark.parametrize("B,H,KV,T,DH,parts", [
    (8, 16, 16, 130, 96, 1), (8, 8, 4, 320, 128, 2), (1, 4, 2, 385, 72, 4), (16, 16, 16, 130, 32, 1), (8, 8, 4, 320, 24, 2),
    (16, 16, 16, 130, 64, 1), (1, 8, 8, 100, 56, 2), (1, 8, 4, 500, 64, 4)])
def test_attention_on_mma_sync_with_and_without_clusters(eng, B, H, KV, T, DH, parts):
    """The head dims and the short or small shapes that stay on attn_mma.cu, by the number of CTAs that share a key tile in dK / dV: the bound of
    the tests above against float64, and the same bits on every run."""
    rng = np.random.default_rng(T + DH)
    q, k, v, do = make(rng, B, H, KV, T, DH, 1)
    scale = 1.0 / np.sqrt(DH)
    runs = run_bf16_attention(eng, q, k, v, do, scale, 0, times=2)
    assert eng.last_variant() == 0x83 + 0x100 * parts
    general = run_bf16_attention(eng, q, k, v, do, scale, 2)[0]
    for n, exact in attention_f64(q, k, v, do, scale).items():
        assert np.array_equal(runs[0][n], runs[1][n]), n
        err = lambda bits: float(np.linalg.norm(E.bf16_bits_to_f32(bits).transpose(0, 2, 1, 3) - exact) / np.linalg.norm(exact))
        assert err(runs[0][n]) <= 1.01 * err(general[n]), (n, err(runs[0][n]), err(general[n]))


@pytest.mark.parametrize("scale", [-0.25, 0.0])
@pytest.mark.parametrize("B,H,KV,T,DH", [(1, 4, 2, 256, 64), (1, 2, 1, 256, 128), (1, 4, 2, 200, 64), (1, 2, 2, 72, 32)])
def test_attention_with_a_scale_that_is_not_positive(eng, B, H, KV, T, DH, scale):
    """Such a scale reverses or flattens the softmax; the tcgen05 kernels mask with -inf in front of the scale and do not take it."""
    rng = np.random.default_rng(T + DH)
    q, k, v, do = make(rng, B, H, KV, T, DH, 1)
    got = run_bf16_attention(eng, q, k, v, do, scale, 0)[0]
    for n, ref in attention_f64(q, k, v, do, scale).items():
        a = E.bf16_bits_to_f32(got[n]).transpose(0, 2, 1, 3)
        assert np.isfinite(a).all(), n
        assert np.abs(a - ref).max() <= (1.5e-2 if n == "o" else 2e-2) * np.abs(ref).max() + 1e-30, n


@pytest.mark.parametrize("B,H,KV,T,DH", [(1, 4, 2, 1000, 64), (1, 3, 1, 130, 64), (2, 8, 4, 256, 32), (1, 2, 2, 385, 128), (1, 2, 1, 200, 96)])
def test_inverse_rotary_of_other_shapes_is_rounded_once(eng, B, H, KV, T, DH):
    """dq and dk that leave the op rotated back (head dims 32, 64, 128; 96 runs the rotary kernel behind the op) against float64: a
    rotation in fp32 leaves the 2-norm error of the unrotated results (1.8e-3: their rounding to bf16 and that of o in the row dots);
    a second rounding would add 1.66e-3 in quadrature, 35 %."""
    rng = np.random.default_rng(T + DH)
    q, k, v, do = make(rng, B, H, KV, T, DH, 1)
    scale = 1.0 / np.sqrt(DH)
    cos, sin = O.rope_tables(T, DH)
    ref = attention_f64(q, k, v, do, scale)
    plain = run_bf16_attention(eng, q, k, v, do, scale, 0)[0]
    ic, isn = put(eng, cos, 0), put(eng, sin, 0)
    t = lambda x: np.ascontiguousarray(x.transpose(0, 2, 1, 3))
    iq, ik, iv, ido = put(eng, t(q), 1), put(eng, t(k), 1), put(eng, t(v), 1), put(eng, t(do), 1)
    io, ilse, iD = eng.alloc(q.size, 2), eng.alloc(B * H * T), eng.alloc(B * H * T + q.size)
    idq, idk, idv = eng.alloc(q.size, 2), eng.alloc(k.size, 2), eng.alloc(k.size, 2)
    eng.launch_count(reset=True)
    eng.run([op(E.ATTN_FWD, a=iq, b=ik, d=iv, c=io, sa=ilse, m=T, n=DH, k=KV, batch=B, tb=H, dt=1, alpha=scale),
             op(E.ATTN_BWD, a=iq, b=ik, d=iv, c=ido, sa=ilse, sb=io, tb=idq, sc=idk, oa=idv, ob=H, oc=iD,
                m=T, n=DH, k=KV, batch=B, dt=1, alpha=scale, beta=float(ic), gamma=float(isn))])
    fused = DH in (32, 64, 128)
    assert eng.launch_count() == (4 if fused else 5)
    c, s = cos.astype(np.float64), sin.astype(np.float64)
    for n, i, heads in (("dq", idq, H), ("dk", idk, KV)):
        g1, g2 = ref[n][..., :DH // 2], ref[n][..., DH // 2:]
        want = np.concatenate([g1 * c + g2 * s, g2 * c - g1 * s], -1)
        err = lambda a, b: float(np.linalg.norm(a - b) / np.linalg.norm(b))
        base = err(E.bf16_bits_to_f32(plain[n]).transpose(0, 2, 1, 3), ref[n])
        assert err(eng.download_bf16(i, (B, T, heads, DH)).transpose(0, 2, 1, 3), want) <= (1.05 if fused else 1.6) * base
    assert eng.device_status() == 0


@pytest.mark.parametrize("rotary", [False, True])
@pytest.mark.parametrize("DH", [64, 128])
@pytest.mark.parametrize("B,H,KV,T,parts", [
    (1, 2, 2, 1024, 4), (2, 2, 1, 512, 4), (3, 12, 4, 512, 2), (3, 8, 4, 256, 2), (1, 10, 10, 512, 2), (3, 30, 10, 768, 1)])       # the first: CTAs with nothing to walk
def test_whole_tile_backward_with_key_tiles_shared_over_a_cluster(eng, B, H, KV, T, DH, parts, rotary):
    """dq, dk and dv against float64, from one CTA to a key tile and from clusters of two and four, plain and rotated back inside.  Bound: bf16 P or dS, result and (in
    the row dots) o, three roundings of at most 2^-9 and 2^-9 / sqrt(3) on average, in quadrature 2.0e-3 in the 2-norm; twice that.  A tile or a pair in the wrong
    place errs by as much as the result."""
    assert eng.lib.eng_attn_tile_parts(B, H, KV, T, DH) == parts
    rng = np.random.default_rng(T + DH + H)
    q, k, v, do = make(rng, B, H, KV, T, DH, 1)
    scale = 1.0 / np.sqrt(DH)
    cos, sin = O.rope_tables(T, DH)
    eng.launch_count(reset=True)
    runs = run_bf16_attention(eng, q, k, v, do, scale, 0, times=2, rotary=(cos, sin) if rotary else ())
    assert eng.launch_count() == 8
    ref = attention_f64(q, k, v, do, scale)
    if rotary:
        c, s = cos.astype(np.float64), sin.astype(np.float64)
        for n in ("dq", "dk"):
            g1, g2 = ref[n][..., :DH // 2], ref[n][..., DH // 2:]
            ref[n] = np.concatenate([g1 * c + g2 * s, g2 * c - g1 * s], -1)
    for n, exact in ref.items():
        got = E.bf16_bits_to_f32(runs[0][n]).transpose(0, 2, 1, 3)
        assert np.linalg.norm(got - exact) <= 4e-3 * np.linalg.norm(exact), n
        assert n == "dq" or np.array_equal(runs[0][n], runs[1][n]), n            # dq is added in the order of arrival
    assert eng.device_status() == 0


@pytest.mark.parametrize("B,H,KV,T", [(20, 8, 8, 128), (10, 8, 8, 512)])
def test_rotary_inside_the_head_dim_128_backward_takes_no_longer_than_a_launch_of_its_own(eng, B, H, KV, T):
    """Many short walks of one CTA each, where the end of a CTA counts (us inside / as a launch of its own on one B200: 30.4 / 33.8 and 62.6 / 66.0; 36 and 70 when each thread rotated a row)."""
    DH = 128
    rng = np.random.default_rng(T)
    q, k, v, do = make(rng, B, H, KV, T, DH, 1)
    t = lambda x: np.ascontiguousarray(x.transpose(0, 2, 1, 3))
    iq, ik, iv, ido = (put(eng, t(x), 1) for x in (q, k, v, do))
    io, ilse, iD = eng.alloc(q.size, 2), eng.alloc(B * H * T), eng.alloc(B * H * T + q.size)
    idq, idk, idv = eng.alloc(q.size, 2), eng.alloc(k.size, 2), eng.alloc(k.size, 2)
    cos, sin = O.rope_tables(T, DH)
    ic, isn = put(eng, cos, 0), put(eng, sin, 0)
    eng.run([op(E.ATTN_FWD, a=iq, b=ik, d=iv, c=io, sa=ilse, m=T, n=DH, k=KV, batch=B, tb=H, dt=1, alpha=DH ** -0.5)])
    bwd = lambda **kw: op(E.ATTN_BWD, a=iq, b=ik, d=iv, c=ido, sa=ilse, sb=io, tb=idq, sc=idk, oa=idv, ob=H, oc=iD, m=T, n=DH, k=KV, batch=B, dt=1, alpha=DH ** -0.5, **kw)
    inside = [bwd(beta=float(ic), gamma=float(isn))] * 40
    apart = [bwd(), op(E.ROPE_BTHD, a=idq, b=ic, d=isn, c=idq, batch=B, m=T, k=H, n=DH, tb=1, sa=idk, sb=idk, sc=KV, dt=1)] * 40
    times = {n: [] for n in ("inside", "apart")}
    for _ in range(6):
        for n, plan in (("inside", inside), ("apart", apart)):
            times[n].append(eng.time_plan(plan, reps=1, flush_l2=False))
    assert min(times["inside"]) <= min(times["apart"]), times
    assert eng.device_status() == 0


@pytest.mark.parametrize("B,H,KV,T,DH", [
    (1, 2, 1, 3, 64), (2, 2, 2, 17, 12), (1, 4, 2, 31, 32), (3, 6, 2, 64, 20), (1, 2, 1, 65, 36), (2, 8, 8, 130, 64), (2, 8, 4, 256, 32), (40, 8, 2, 100, 48), (1, 3, 3, 449, 16),
    (2, 16, 16, 333, 64)])
def test_fp32_attention_of_head_dims_up_to_64(eng, B, H, KV, T, DH):
    """Rows that end inside a lane's four, a warp's sixteen and a block's 64, heads narrower than the columns of a tile, one CTA to a block and clusters of up to eight (some with
    no tile): o, lse, dq, dk and dv against float64 within the bound of the fp32 tests above, nothing behind the last row, the same bits on every run.  (With one
    token dq and dk are zero, the difference of two equal sums, and a bound by the largest element says nothing.)"""
    rng = np.random.default_rng(T + DH)
    q, k, v, do = make(rng, B, H, KV, T, DH, 0)
    scale = 1.0 / np.sqrt(DH)
    t = lambda x: np.ascontiguousarray(x.transpose(0, 2, 1, 3))
    iq, ik, iv, ido = put(eng, t(q), 0), put(eng, t(k), 0), put(eng, t(v), 0), put(eng, t(do), 0)
    guard = 256
    out = {n: (eng.alloc(a.size + guard), a.shape[1], a.size) for n, a in (("o", q), ("dq", q), ("dk", k), ("dv", k))}
    for i, _, n in out.values():
        eng.upload(i, np.full(n + guard, 7.0, np.float32))
    ilse, iD = eng.alloc(B * H * T), eng.alloc(B * H * T)
    runs = []
    for _ in range(2):
        eng.run([op(E.ATTN_FWD, a=iq, b=ik, d=iv, c=out["o"][0], sa=ilse, m=T, n=DH, k=KV, batch=B, tb=H, dt=0, alpha=scale)])
        assert eng.last_variant() == 0x84
        eng.run([op(E.ATTN_BWD, a=iq, b=ik, d=iv, c=ido, sa=ilse, sb=out["o"][0], tb=out["dq"][0], sc=out["dk"][0], oa=out["dv"][0], ob=H, oc=iD, m=T, n=DH, k=KV,
                    batch=B, dt=0, alpha=scale)])
        assert eng.last_variant() == 0x85
        runs.append({n: eng.download(i, (sz + guard,)) for n, (i, _, sz) in out.items()})
    for n, ref in attention_f64(q, k, v, do, scale).items():
        heads, sz = out[n][1:]
        got = runs[0][n][:sz].reshape(B, T, heads, DH).transpose(0, 2, 1, 3)
        assert np.abs(got - ref).max() <= 2e-5 * np.abs(ref).max() + 1e-30, n
        assert np.array_equal(runs[0][n], runs[1][n]) and np.all(runs[0][n][sz:] == 7.0), n
    assert np.abs(eng.download(ilse, (B, H, T)) - O.attention_fwd(q, k, v, scale)[1]).max() <= 2e-5
    assert eng.device_status() == 0
