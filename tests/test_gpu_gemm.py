"""GEMM op (kinds GEMM / GEMM_SB / GEMM_EX) on the GPU against numpy: the three
operand layouts the plan uses (tb 0/1/2, axis/engine.py:47), fp32 and bf16
storage, bf16-in/fp32-out weight gradients, alpha/beta epilogues, offsets and
strided batches, tile tails, and tensor-core path vs general path agreement."""
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


def run_gemm(eng, rng, m, n, k, tb, dt, alpha=0.0, beta=0.0, addend=False, fallback=0):
    in_bf, out_bf = dt >= 1, dt == 1
    sha = (k, m) if tb == 2 else (m, k)
    shb = (n, k) if tb == 1 else (k, n)
    A = rng.standard_normal(sha).astype(np.float32)
    B = rng.standard_normal(shb).astype(np.float32)
    C0 = rng.standard_normal((m, n)).astype(np.float32)
    if in_bf:
        A, B = bf(A), bf(B)
    if out_bf:
        C0 = bf(C0)
    ia, ib = put(eng, A, in_bf), put(eng, B, in_bf)
    ic = put(eng, C0, out_bf)
    idd = put(eng, C0, out_bf) if addend else -1
    if addend:
        eng.upload_bf16(ic, np.zeros((m, n), np.float32)) if out_bf else eng.upload(ic, np.zeros((m, n), np.float32))
    eng.set_fallback(fallback)
    kind = E.GEMM_EX if addend else E.GEMM_SB
    eng.run([op(kind, a=ia, b=ib, c=ic, d=idd, m=m, n=n, k=k, batch=1, tb=tb, dt=dt, alpha=alpha, beta=beta)])
    eng.set_fallback(0)
    got = eng.download_bf16(ic, (m, n)) if out_bf else eng.download(ic, (m, n))
    Aop = A.T if tb == 2 else A
    Bop = B.T if tb == 1 else B
    ref = (alpha if alpha != 0.0 else 1.0) * (Aop.astype(np.float64) @ Bop.astype(np.float64)) + beta * C0
    return got, ref.astype(np.float32)


def check(got, ref, out_bf, k):
    scale = np.abs(ref).max() + 1e-6
    err = np.abs(got - ref).max() / scale
    lim = 6e-3 if out_bf else 3e-6 * max(1.0, np.sqrt(k) / 4)
    assert err <= lim, (err, lim)


@pytest.mark.parametrize("tb", [0, 1, 2])
@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (5, 7, 3), (64, 64, 16), (100, 130, 70), (257, 96, 33)])
def test_fp32_gemm_is_true_fp32(eng, tb, m, n, k):
    rng = np.random.default_rng(m * n + k)
    got, ref = run_gemm(eng, rng, m, n, k, tb, 0)
    check(got, ref, False, k)
    got, ref = run_gemm(eng, rng, m, n, k, tb, 0, alpha=0.5, beta=1.0)
    check(got, ref, False, k)


@pytest.mark.parametrize("tb", [0, 1, 2])
@pytest.mark.parametrize("dt", [1, 2])
@pytest.mark.parametrize("m,n,k", [(128, 128, 64), (256, 256, 128), (384, 512, 192), (200, 136, 72),
                                   (128, 264, 1000), (1000, 128, 64)])
def test_bf16_tensor_core_gemm(eng, tb, dt, m, n, k):
    if tb == 2 and m % 8:
        pytest.skip("M-major operand needs m % 8 == 0 for the TMA path")
    rng = np.random.default_rng(m + n + k + tb)
    got, ref = run_gemm(eng, rng, m, n, k, tb, dt)
    check(got, ref, dt == 1, k)
    assert eng.device_status() == 0


@pytest.mark.parametrize("tb", [0, 1, 2])
def test_bf16_epilogues_and_addend(eng, tb):
    rng = np.random.default_rng(tb)
    for dt in (1, 2):
        got, ref = run_gemm(eng, rng, 256, 384, 128, tb, dt, alpha=2.0, beta=1.0)
        check(got, ref, dt == 1, 128)
        got, ref = run_gemm(eng, rng, 256, 384, 128, tb, dt, beta=1.0, addend=True)
        check(got, ref, dt == 1, 128)


@pytest.mark.parametrize("tb", [0, 1, 2])
@pytest.mark.parametrize("dt", [1, 2])
@pytest.mark.parametrize("m,n,k", [(520, 776, 320), (256, 264, 64), (1032, 256, 2112)])
def test_paired_kernel_staged_output(eng, tb, dt, m, n, k):
    """Paired-CTA kernel forced (mask 8): output pieces staged in shared memory and written by TMA
    stores clipped at ragged edges; in-place accumulation and a separate addend arrive by TMA loads;
    the long-k shape also runs the split-K workspace through the same stores."""
    rng = np.random.default_rng(m + n + k + tb + dt)
    got, ref = run_gemm(eng, rng, m, n, k, tb, dt, fallback=8)
    check(got, ref, dt == 1, k)
    got, ref = run_gemm(eng, rng, m, n, k, tb, dt, alpha=0.5, beta=1.0, fallback=8)
    check(got, ref, dt == 1, k)
    got, ref = run_gemm(eng, rng, m, n, k, tb, dt, beta=-2.0, addend=True, fallback=8)
    check(got, ref, dt == 1, k)
    assert eng.device_status() == 0


@pytest.mark.parametrize("tb", [0, 1, 2])
def test_tensor_core_and_general_path_agree(eng, tb):
    for dt in (1, 2):
        a = run_gemm(eng, np.random.default_rng(9), 256, 256, 256, tb, dt)[0]
        b = run_gemm(eng, np.random.default_rng(9), 256, 256, 256, tb, dt, fallback=1)[0]
        assert np.abs(a - b).max() <= (2e-2 if dt == 1 else 1e-3) * np.abs(b).max()


@pytest.mark.parametrize("dt", [0, 1])
def test_small_and_unaligned_bf16_and_batched_offsets(eng, dt):
    rng = np.random.default_rng(5)
    for (m, n, k, tb) in [(3, 5, 7, 0), (130, 16, 136, 0), (16, 130, 130, 2), (130, 136, 16, 1), (129, 131, 67, 1)]:
        got, ref = run_gemm(eng, rng, m, n, k, tb, dt)
        check(got, ref, dt == 1, k)
    # strided batch with element offsets, as the tiled attention plan issues them
    batch, qt, kl, DH, T, rep = 4, 8, 24, 16, 32, 2
    q = rng.standard_normal((batch, rep, T, DH)).astype(np.float32)
    kk = rng.standard_normal((batch, T, DH)).astype(np.float32)
    if dt:
        q, kk = bf(q), bf(kk)
    iq, ik, ic = put(eng, q, dt), put(eng, kk, dt), eng.alloc(batch * qt * kl)
    j, qs = 1, 16
    eng.run([op(E.GEMM_SB, a=iq, b=ik, c=ic, m=qt, k=DH, n=kl, batch=batch, tb=1, sa=rep * T * DH, sb=T * DH,
                sc=qt * kl, oa=(j * T + qs) * DH, dt=dt, alpha=0.25)])
    ref = 0.25 * np.einsum("bqd,bkd->bqk", q[:, j, qs:qs + qt], kk[:, :kl])
    got = eng.download_bf16(ic, ref.shape) if dt else eng.download(ic, ref.shape)
    check(got, ref, dt == 1, DH)


@pytest.mark.parametrize("dt", [0, 1, 2])
@pytest.mark.parametrize("tb", [0, 1, 2])
@pytest.mark.parametrize("count", [2, 3])
def test_grouped_gemm_shared_input(eng, dt, tb, count):
    """GEMM_GROUP mode 1: one input, several outputs with their own widths (ragged ones included)."""
    rng = np.random.default_rng(10 * tb + count + dt)
    m, k, ns = 520, 320, (520, 264, 136)[:count]
    in_bf, out_bf = dt >= 1, dt == 1
    A = rng.standard_normal((k, m) if tb == 2 else (m, k)).astype(np.float32)
    Bs = [rng.standard_normal((n, k) if tb == 1 else (k, n)).astype(np.float32) for n in ns]
    if in_bf:
        A, Bs = bf(A), [bf(b) for b in Bs]
    ia = put(eng, A, in_bf)
    ib = [put(eng, b, in_bf) for b in Bs] + [0]
    ic = [eng.alloc(m * n, 2 if out_bf else 4) for n in ns] + [0]
    nn = list(ns) + [0]
    eng.run([op(E.GEMM_GROUP, a=ia, b=ib[0], sa=ib[1], sb=ib[2], c=ic[0], d=ic[1], sc=ic[2], m=m, k=k,
                n=nn[0], oa=nn[1], ob=nn[2], batch=count, oc=1, tb=tb, dt=dt, alpha=0.5)])
    Aop = A.T if tb == 2 else A
    for g, n in enumerate(ns):
        got = eng.download_bf16(ic[g], (m, n)) if out_bf else eng.download(ic[g], (m, n))
        Bop = Bs[g].T if tb == 1 else Bs[g]
        check(got, (0.5 * (Aop.astype(np.float64) @ Bop.astype(np.float64))).astype(np.float32), out_bf, k)
    assert eng.device_status() == 0


@pytest.mark.parametrize("dt", [0, 1, 2])
@pytest.mark.parametrize("tb", [0, 1, 2])
@pytest.mark.parametrize("count", [2, 3])
def test_grouped_gemm_summed_segments(eng, dt, tb, count):
    """GEMM_GROUP mode 2: one output accumulated over K-segments of different depths (one not a multiple
    of the 64-wide k-block)."""
    rng = np.random.default_rng(100 + 10 * tb + count + dt)
    m, n, ks = 520, 392, (320, 136, 200)[:count]
    in_bf, out_bf = dt >= 1, dt == 1
    As = [rng.standard_normal((k, m) if tb == 2 else (m, k)).astype(np.float32) for k in ks]
    Bs = [rng.standard_normal((n, k) if tb == 1 else (k, n)).astype(np.float32) for k in ks]
    if in_bf:
        As, Bs = [bf(a) for a in As], [bf(b) for b in Bs]
    ia = [put(eng, a, in_bf) for a in As] + [0]
    ib = [put(eng, b, in_bf) for b in Bs] + [0]
    ic = eng.alloc(m * n, 2 if out_bf else 4)
    kk = list(ks) + [0]
    eng.run([op(E.GEMM_GROUP, c=ic, a=ia[0], sa=ia[1], sb=ia[2], b=ib[0], d=ib[1], sc=ib[2], m=m, n=n,
                k=kk[0], oa=kk[1], ob=kk[2], batch=count, oc=2, tb=tb, dt=dt)])
    ref = np.zeros((m, n), np.float64)
    for a, b_ in zip(As, Bs):
        ref += (a.T if tb == 2 else a).astype(np.float64) @ (b_.T if tb == 1 else b_).astype(np.float64)
    got = eng.download_bf16(ic, (m, n)) if out_bf else eng.download(ic, (m, n))
    check(got, ref.astype(np.float32), out_bf, sum(ks))
    assert eng.device_status() == 0


@pytest.mark.parametrize("dt", [0, 1, 2])
@pytest.mark.parametrize("tb", [0, 1, 2])
def test_grouped_gemm_independent_problems(eng, dt, tb):
    """GEMM_GROUP mode 3: two problems with their own operands, heights and widths, one depth."""
    rng = np.random.default_rng(300 + 10 * tb + dt)
    k, ms, ns = 328, (776, 264), (392, 520)
    in_bf, out_bf = dt >= 1, dt == 1
    As = [rng.standard_normal((k, m) if tb == 2 else (m, k)).astype(np.float32) for m in ms]
    Bs = [rng.standard_normal((n, k) if tb == 1 else (k, n)).astype(np.float32) for n in ns]
    if in_bf:
        As, Bs = [bf(a) for a in As], [bf(b) for b in Bs]
    ia = [put(eng, a, in_bf) for a in As]
    ib = [put(eng, b, in_bf) for b in Bs]
    ic = [eng.alloc(m * n, 2 if out_bf else 4) for m, n in zip(ms, ns)]
    eng.run([op(E.GEMM_GROUP, a=ia[0], sa=ia[1], b=ib[0], sb=ib[1], c=ic[0], d=ic[1], m=ms[0], oa=ms[1],
                n=ns[0], ob=ns[1], k=k, batch=2, oc=3, tb=tb, dt=dt)])
    for g in range(2):
        got = eng.download_bf16(ic[g], (ms[g], ns[g])) if out_bf else eng.download(ic[g], (ms[g], ns[g]))
        ref = (As[g].T if tb == 2 else As[g]).astype(np.float64) @ (Bs[g].T if tb == 1 else Bs[g]).astype(np.float64)
        check(got, ref.astype(np.float32), out_bf, k)
    assert eng.device_status() == 0


@pytest.mark.parametrize("dt", [0, 1])
@pytest.mark.parametrize("m,n,k", [(520, 392, 320), (256, 128, 64), (1032, 1000, 136)])
def test_grouped_gemm_swiglu_pair(eng, dt, m, n, k):
    """GEMM_GROUP mode 4: gate and up projections with h = silu(g) * u written by the same launch (bf16);
    the fp32 plan runs the unfused sequence behind the same op."""
    rng = np.random.default_rng(m + n + k + dt)
    A = rng.standard_normal((m, k)).astype(np.float32) * 0.5
    Wg = rng.standard_normal((k, n)).astype(np.float32) * 0.2
    Wu = rng.standard_normal((k, n)).astype(np.float32) * 0.2
    if dt:
        A, Wg, Wu = bf(A), bf(Wg), bf(Wu)
    ia, ig, iu = put(eng, A, dt), put(eng, Wg, dt), put(eng, Wu, dt)
    og, ou, oh = (eng.alloc(m * n, 2 if dt else 4) for _ in range(3))
    eng.run([op(E.GEMM_GROUP, a=ia, b=ig, sa=iu, c=og, d=ou, sc=oh, m=m, n=n, k=k, batch=2, oc=4, dt=dt)])
    g = A.astype(np.float64) @ Wg.astype(np.float64)
    u = A.astype(np.float64) @ Wu.astype(np.float64)
    h = g / (1.0 + np.exp(-g)) * u
    get_ = (lambda i: eng.download_bf16(i, (m, n))) if dt else (lambda i: eng.download(i, (m, n)))
    check(get_(og), g.astype(np.float32), dt == 1, k)
    check(get_(ou), u.astype(np.float32), dt == 1, k)
    check(get_(oh), h.astype(np.float32), dt == 1, k)
    assert eng.device_status() == 0


@pytest.mark.parametrize("fallback", [0, 1, 8])
def test_grouped_projection_with_rotary_in_the_epilogue(eng, fallback):
    """GEMM_GROUP mode 1 with gamma > 0: q and k leave the launch rotated, v does not.  fallback 0: the small-product
    kernel (mask 8: the paired-CTA one) rotates in its epilogue (fp32 accumulators, one rounding); fallback 1: general GEMMs, then the
    rotary kernel."""
    rng = np.random.default_rng(5)
    B_, T, D, H, KV = 2, 256, 192, 6, 2
    N = B_ * T
    bf = lambda a: E.bf16_bits_to_f32(E.f32_to_bf16_bits(a))
    x = bf(rng.standard_normal((N, D)).astype(np.float32))
    wq, wk, wv = (bf(rng.standard_normal((D, w)).astype(np.float32) * 0.1) for w in (H * 64, KV * 64, KV * 64))
    cos, sin = O.rope_tables(T, 64)

    def put(a, bf16=True):
        i = eng.alloc(a.size, 2 if bf16 else 4)
        eng.upload_bf16(i, a) if bf16 else eng.upload(i, a)
        return i
    ix, iq, ik, iv = put(x), put(wq), put(wk), put(wv)
    ic, isn = put(cos, False), put(sin, False)
    oq, ok_, ov = eng.alloc(N * H * 64, 2), eng.alloc(N * KV * 64, 2), eng.alloc(N * KV * 64, 2)
    eng.set_fallback(fallback)
    eng.launch_count(reset=True)
    eng.run([op(E.GEMM_GROUP, a=ix, b=iq, sa=ik, sb=iv, c=oq, d=ok_, sc=ov, m=N, k=D, n=H * 64, oa=KV * 64, ob=KV * 64,
                batch=3, oc=1, dt=1, beta=float(ic), gamma=float(isn))])
    launches = eng.launch_count()
    eng.set_fallback(0)
    assert launches == (4 if fallback == 1 else 1)
    assert fallback == 1 or eng.last_variant() == (0x23 if fallback else 0x26)
    rot = lambda y, heads: O.rope_fwd(y.reshape(B_, T, heads, 64).transpose(0, 2, 1, 3), cos, sin).transpose(0, 2, 1, 3).reshape(N, heads * 64)
    q_ref, k_ref, v_ref = rot(x @ wq, H), rot(x @ wk, KV), x @ wv
    for got, ref in ((eng.download_bf16(oq, (N, H * 64)), q_ref), (eng.download_bf16(ok_, (N, KV * 64)), k_ref),
                     (eng.download_bf16(ov, (N, KV * 64)), v_ref)):
        assert np.abs(got - ref).max() <= 1.2e-2 * np.abs(ref).max()
    assert eng.device_status() == 0


@pytest.mark.parametrize("dt", [0, 1])
@pytest.mark.parametrize("tb", [0, 1])
@pytest.mark.parametrize("count", [2, 3])
def test_grouped_gemm_shared_input_with_a_low_rank_term_per_output(eng, dt, tb, count):
    """GEMM_XSEG before GEMM_GROUP mode 1: C_g = alpha * (A B_g + A'_g B'_g) — an adapter's rank-16 product as a
    K-segment of its projection's launch; the variant number tells that the grouped kernel served it in bf16."""
    rng = np.random.default_rng(500 + 10 * tb + count + dt)
    m, k, r, ns = 520, 320, 16, (520, 264, 136)[:count]
    mk = lambda sh: bf(rng.standard_normal(sh).astype(np.float32)) if dt else rng.standard_normal(sh).astype(np.float32)
    A = mk((m, k))
    Bs = [mk((n, k) if tb == 1 else (k, n)) for n in ns]
    XAs = [mk((m, r)) for _ in ns]
    XBs = [mk((n, r) if tb == 1 else (r, n)) for n in ns]
    ia = put(eng, A, dt)
    ib = [put(eng, b, dt) for b in Bs] + [0]
    xa = [put(eng, a, dt) for a in XAs] + [0]
    xb = [put(eng, b, dt) for b in XBs] + [0]
    ic = [eng.alloc(m * n, 2 if dt else 4) for n in ns] + [0]
    nn = list(ns) + [0]
    eng.launch_count(reset=True)
    eng.run([op(E.GEMM_XSEG, a=xa[0], b=xa[1], d=xa[2], sa=xb[0], sb=xb[1], sc=xb[2], k=r, batch=count),
             op(E.GEMM_GROUP, a=ia, b=ib[0], sa=ib[1], sb=ib[2], c=ic[0], d=ic[1], sc=ic[2], m=m, k=k,
                n=nn[0], oa=nn[1], ob=nn[2], batch=count, oc=1, tb=tb, dt=dt, alpha=0.5)])
    if dt:
        assert eng.launch_count() == 1                       # one grouped launch, nothing run one by one
    for g, n in enumerate(ns):
        got = eng.download_bf16(ic[g], (m, n)) if dt else eng.download(ic[g], (m, n))
        Bop = Bs[g].T if tb == 1 else Bs[g]
        XBop = XBs[g].T if tb == 1 else XBs[g]
        ref = 0.5 * (A.astype(np.float64) @ Bop.astype(np.float64) + XAs[g].astype(np.float64) @ XBop.astype(np.float64))
        check(got, ref.astype(np.float32), dt == 1, k + r)
    assert eng.device_status() == 0


@pytest.mark.parametrize("dt", [0, 1])
@pytest.mark.parametrize("tb", [0, 1])
@pytest.mark.parametrize("count,extra,addend", [(3, 3, False), (1, 1, True), (2, 2, True), (3, 1, False)])
@pytest.mark.parametrize("mask", [0, 8])
def test_grouped_gemm_up_to_six_segments_and_an_addend(eng, mask, dt, tb, count, extra, addend):
    """GEMM_XSEG before GEMM_GROUP mode 2: further K-segments (depth 16) behind the op's own, and a residual addend:
    C = sum_s A_s B_s + D."""
    rng = np.random.default_rng(600 + 10 * tb + 3 * count + extra + dt)
    m, n, r, ks = 520, 392, 16, (320, 136, 200)[:count]
    mk = lambda sh: bf(rng.standard_normal(sh).astype(np.float32)) if dt else rng.standard_normal(sh).astype(np.float32)
    As = [mk((m, k)) for k in ks] + [mk((m, r)) for _ in range(extra)]
    Bs = [mk((n, k) if tb == 1 else (k, n)) for k in ks] + [mk((n, r) if tb == 1 else (r, n)) for _ in range(extra)]
    D = mk((m, n))
    ia = [put(eng, a, dt) for a in As[:count]] + [0, 0]
    ib = [put(eng, b, dt) for b in Bs[:count]] + [0, 0]
    xa = [put(eng, a, dt) for a in As[count:]] + [0, 0]
    xb = [put(eng, b, dt) for b in Bs[count:]] + [0, 0]
    idd = put(eng, D, dt) if addend else 0
    ic = eng.alloc(m * n, 2 if dt else 4)
    kk = list(ks) + [0, 0]
    eng.set_fallback(mask)
    eng.launch_count(reset=True)
    eng.run([op(E.GEMM_XSEG, a=xa[0], b=xa[1], d=xa[2], sa=xb[0], sb=xb[1], sc=xb[2], k=r, batch=extra, c=idd, beta=1.0),
             op(E.GEMM_GROUP, c=ic, a=ia[0], sa=ia[1], sb=ia[2], b=ib[0], d=ib[1], sc=ib[2], m=m, n=n,
                k=kk[0], oa=kk[1], ob=kk[2], batch=count, oc=2, tb=tb, dt=dt)])
    eng.set_fallback(0)
    if dt:
        assert eng.launch_count() == 1 and eng.last_variant() == (0x23 if mask else 0x26)
    ref = D.astype(np.float64) if addend else np.zeros((m, n), np.float64)
    for a, b_ in zip(As, Bs):
        ref = ref + a.astype(np.float64) @ (b_.T if tb == 1 else b_).astype(np.float64)
    got = eng.download_bf16(ic, (m, n)) if dt else eng.download(ic, (m, n))
    check(got, ref.astype(np.float32), dt == 1, sum(ks) + r * extra)
    assert eng.device_status() == 0


def test_extra_operands_are_refused_where_they_have_no_meaning(eng):
    """A GEMM_XSEG whose count differs from the mode-1 group's, or before a mode-3 group, is an error, and the pending
    operands do not leak into a later group."""
    rng = np.random.default_rng(7)
    m, k, n, r = 256, 64, 64, 16
    A, B = bf(rng.standard_normal((m, k)).astype(np.float32)), bf(rng.standard_normal((k, n)).astype(np.float32))
    ia, ib, ic, id_ = put(eng, A, 1), put(eng, B, 1), eng.alloc(m * n, 2), eng.alloc(m * n, 2)
    xa, xb = put(eng, bf(rng.standard_normal((m, r)).astype(np.float32)), 1), put(eng, bf(rng.standard_normal((r, n)).astype(np.float32)), 1)
    grp = op(E.GEMM_GROUP, a=ia, b=ib, sa=ib, c=ic, d=id_, m=m, k=k, n=n, oa=n, batch=2, oc=1, dt=1)
    with pytest.raises(RuntimeError):
        eng.run([op(E.GEMM_XSEG, a=xa, sa=xb, k=r, batch=1), grp])
    eng.run([grp])                                   # the refused operands are gone
    got = eng.download_bf16(ic, (m, n))
    check(got, (A.astype(np.float64) @ B.astype(np.float64)).astype(np.float32), True, k)


@pytest.mark.parametrize("layout", [0, 1])
@pytest.mark.parametrize("R", [8, 16, 32])
def test_adapter_gradients_stream_kernel(eng, layout, R):
    """LORA_GRAD: alpha * X_g^T S_g for three products (ragged widths and token count), written at offsets of one fp32
    buffer as [F, R] or [R, F]; bit-identical on a second run (fixed summation order)."""
    rng = np.random.default_rng(800 + layout + R)
    N, Fs = 1000, (520, 264, 1536)
    Xs = [bf(rng.standard_normal((N, F)).astype(np.float32)) for F in Fs]
    Ss = [bf(rng.standard_normal((N, R)).astype(np.float32)) for _ in Fs]
    ix = [put(eng, x, 1) for x in Xs]
    is_ = [put(eng, s_, 1) for s_ in Ss]
    offs = [64, 64 + Fs[0] * R + 8, 64 + Fs[0] * R + 8 + Fs[1] * R + 8]
    total = offs[2] + Fs[2] * R + 64
    out = eng.alloc(total)
    eng.upload(out, np.full(total, 7.0, np.float32))
    plan = [op(E.LORA_GRAD, a=ix[0], sa=ix[1], sb=ix[2], b=is_[0], d=is_[1], sc=is_[2], c=out, oa=offs[0], ob=offs[1],
               oc=offs[2], n=Fs[0], k=Fs[1], tb=Fs[2], m=N, batch=3, gamma=float(R), beta=float(layout), alpha=0.5, dt=1)]
    eng.run(plan)
    assert eng.last_variant() == 0x60                         # the streaming kernel, not the GEMM path
    got = eng.download(out, total)
    eng.run(plan)
    assert np.array_equal(got, eng.download(out, total))
    touched = np.zeros(total, bool)
    for g, F in enumerate(Fs):
        ref = 0.5 * (Xs[g].astype(np.float64).T @ Ss[g].astype(np.float64))
        ref = ref.T if layout else ref
        seg = got[offs[g]:offs[g] + F * R].reshape(ref.shape)
        assert np.abs(seg - ref).max() <= 2e-5 * np.abs(ref).max() + 1e-4
        touched[offs[g]:offs[g] + F * R] = True
    assert np.all(got[~touched] == 7.0)                       # nothing outside the three outputs is written
    # the GEMM path (library fallback switch) gives the same numbers within fp32 summation order
    eng.set_fallback(1)
    eng.run(plan)
    eng.set_fallback(0)
    assert np.abs(eng.download(out, total) - got)[touched].max() <= 1e-3 * np.abs(got[touched]).max()
    assert eng.device_status() == 0


@pytest.mark.parametrize("tb", [0, 1])
@pytest.mark.parametrize("R", [8, 16, 32])
def test_adapter_skinny_products_stream_kernel(eng, tb, R):
    """LORA_PROJ: out_g [N, R] = alpha * X_g W_g (W [F, R]) or X_g W_g^T (W [R, F]) for three adapters at once, ragged token
    count and widths (one narrower than a 256-column piece, one of several pieces)."""
    rng = np.random.default_rng(900 + tb + R)
    N, Fs = 1000, (520, 136, 1536)
    Xs = [bf(rng.standard_normal((N, F)).astype(np.float32)) for F in Fs]
    Ws = [bf(rng.standard_normal((R, F) if tb else (F, R)).astype(np.float32) * 0.1) for F in Fs]
    ix, iw = [put(eng, x, 1) for x in Xs], [put(eng, w, 1) for w in Ws]
    io = [eng.alloc(N * R + 64, 2) for _ in Fs]
    for o_ in io:
        eng.upload_bf16(o_, np.full(N * R + 64, 3.0, np.float32))
    plan = [op(E.LORA_PROJ, a=ix[0], sa=ix[1], sb=ix[2], b=iw[0], d=iw[1], sc=iw[2], c=io[0], oa=io[1], ob=io[2],
               n=Fs[0], k=Fs[1], oc=Fs[2], m=N, batch=3, tb=tb, gamma=float(R), alpha=2.0, dt=1)]
    eng.launch_count(reset=True)
    eng.run(plan)
    assert eng.last_variant() == 0x62 and eng.launch_count() == 1
    for g, F in enumerate(Fs):
        got = eng.download_bf16(io[g], (N * R + 64,))
        ref = 2.0 * (Xs[g].astype(np.float64) @ (Ws[g].T if tb else Ws[g]).astype(np.float64))
        check(got[:N * R].reshape(N, R), ref.astype(np.float32), True, F)
        assert np.all(got[N * R:] == 3.0)
    # one shared input (the u_g = x A_g of projections of one input), against the GEMM path
    plan2 = [op(E.LORA_PROJ, a=ix[2], b=iw[2], d=iw[2], c=io[0], oa=io[1], n=Fs[2], k=Fs[2], m=N, batch=2, tb=tb,
                gamma=float(R), dt=1)]
    eng.run(plan2)
    a0, a1 = eng.download_bf16(io[0], (N, R)), eng.download_bf16(io[1], (N, R))
    assert np.array_equal(a0, a1)
    eng.set_fallback(1)
    eng.run(plan2)
    eng.set_fallback(0)
    check(eng.download_bf16(io[0], (N, R)), a0, True, Fs[2])
    assert eng.device_status() == 0


def test_adapter_gradients_noted_and_run_as_one_launch(eng):
    """LORA_GRAD with batch < 0 only notes its products; batch = 0 runs all of them (both layouts mixed) as one launch pair."""
    rng = np.random.default_rng(77)
    N, R, Fs = 777, 16, (264, 520, 136, 1032)
    Xs = [bf(rng.standard_normal((N, F)).astype(np.float32)) for F in Fs]
    Ss = [bf(rng.standard_normal((N, R)).astype(np.float32)) for _ in Fs]
    ix, is_ = [put(eng, x, 1) for x in Xs], [put(eng, s_, 1) for s_ in Ss]
    offs = list(np.cumsum([0] + [F * R for F in Fs]))
    out = eng.alloc(int(offs[-1]))
    eng.upload(out, np.zeros(int(offs[-1]), np.float32))
    eng.launch_count(reset=True)
    eng.run([op(E.LORA_GRAD, a=ix[0], sa=ix[1], b=is_[0], d=is_[1], c=out, oa=int(offs[0]), ob=int(offs[1]), n=Fs[0], k=Fs[1],
                m=N, batch=-2, gamma=float(R), dt=1),
             op(E.LORA_GRAD, a=ix[2], sa=ix[3], b=is_[2], d=is_[3], c=out, oa=int(offs[2]), ob=int(offs[3]), n=Fs[2], k=Fs[3],
                m=N, batch=-2, gamma=float(R), beta=1.0, dt=1)])
    assert eng.launch_count() == 0 and np.all(eng.download(out, int(offs[-1])) == 0)      # nothing has run yet
    eng.run([op(E.LORA_GRAD, batch=0)])
    assert eng.launch_count() == 2 and eng.last_variant() == 0x60
    got = eng.download(out, int(offs[-1]))
    for g, F in enumerate(Fs):
        ref = Xs[g].astype(np.float64).T @ Ss[g].astype(np.float64)
        ref = ref.T if g >= 2 else ref
        seg = got[offs[g]:offs[g + 1]].reshape(ref.shape)
        assert np.abs(seg - ref).max() <= 2e-5 * np.abs(ref).max() + 1e-4
    eng.run([op(E.LORA_GRAD, batch=0)])              # an empty set is a no-op
    assert eng.launch_count() == 2 and eng.device_status() == 0


@pytest.mark.parametrize("m,n,k,batch", [
    (1, 1, 1, 1), (31, 33, 65, 1), (512, 256, 256, 1), (256, 256, 1024, 1), (64, 48, 2048, 1), (32, 32, 250, 3),   # 32 x 32 and 64 x 32 tiles, split 1 to 8
    (700, 820, 100, 1), (830, 770, 33, 1), (200, 200, 72, 12),                                                     # 32 x 32 tiles, more than run at once
    (1664, 1540, 96, 1), (1601, 1603, 17, 1)])                                                                     # 64 x 64 tiles
@pytest.mark.parametrize("tb", [0, 1, 2])
def test_fp32_gemm_tiles_and_splits(eng, m, n, k, batch, tb):
    """fp32 GEMM over its sizes, with remainders in each dimension, pitches that do and do not allow 16-byte copies, and
    the depth split over a cluster (each tile by name: `test_fp32_products_on_the_tiles_they_are_cut_into`).  Limit: k products of N(0,1) pairs summed in fp32 in any order err by about
    2^-24 sqrt(k) of the result's rms sqrt(k) per element; ten times that covers the largest of 2.6 million elements."""
    rng = np.random.default_rng(m * 7 + n * 3 + k + tb)
    a = rng.standard_normal((batch, k, m) if tb == 2 else (batch, m, k)).astype(np.float32)
    b = rng.standard_normal((batch, n, k) if tb == 1 else (batch, k, n)).astype(np.float32)
    d = rng.standard_normal((batch, m, n)).astype(np.float32)
    ia, ib, ic, idd = eng.new_tensor(a), eng.new_tensor(b), eng.alloc(d.size + 64), eng.new_tensor(d)
    eng.upload(ic, np.full(d.size + 64, 7.0, np.float32))
    plan = [op(E.GEMM_EX, a=ia, b=ib, c=ic, d=idd, m=m, n=n, k=k, batch=batch, tb=tb, sa=m * k, sb=k * n, sc=m * n, alpha=0.5, beta=-2.0)]
    eng.run(plan)
    out = eng.download(ic, d.size + 64)
    assert np.all(out[d.size:] == 7.0)
    a64 = a.astype(np.float64).transpose(0, 2, 1) if tb == 2 else a.astype(np.float64)
    b64 = b.astype(np.float64).transpose(0, 2, 1) if tb == 1 else b.astype(np.float64)
    ref = 0.5 * (a64 @ b64) - 2.0 * d
    assert np.abs(out[:d.size].reshape(ref.shape) - ref).max() <= 10 * 2.0 ** -24 * (k + 4)
    eng.run(plan)
    assert np.array_equal(out, eng.download(ic, d.size + 64))       # run-to-run identical


@pytest.mark.parametrize("m,n,k,batch,cuts", [           # cuts of A B, A B^T, A^T B
    (1100, 1100, 200, 1, [(64, 64, 8, 1)] * 3), (1093, 1101, 267, 1, [(64, 64, 4, 1)] * 2 + [(64, 64, 8, 1)]), (1613, 1101, 267, 1, [(64, 64, 4, 1), (64, 64, 8, 1), (64, 64, 4, 1)]), (1032, 2085, 13, 1, [(128, 128, 8, 1)] * 3), (200, 200, 72, 19, [(64, 64, 8, 1), (64, 64, 4, 1), (64, 64, 8, 1)]),
    (1100, 900, 24, 1, [(64, 64, 4, 1)] * 3), (1085, 907, 31, 1, [(64, 64, 4, 1)] * 3), (700, 1050, 451, 1, [(64, 64, 4, 1)] * 2 + [(32, 32, 4, 1)]),
    (512, 256, 256, 1, [(64, 32, 8, 4)] * 3), (517, 218, 251, 1, [(32, 32, 4, 2)] + [(64, 32, 8, 4)] * 2), (517, 250, 251, 1, [(32, 32, 4, 2)] * 3), (1528, 1404, 76, 1, [(64, 64, 4, 1)] * 3), (523, 781, 300, 1, [(64, 32, 8, 1)] * 3), (120, 424, 1960, 1, [(64, 32, 8, 8)] * 3),
    (31, 33, 65, 1, [(32, 32, 4, 1)] * 3), (90, 70, 1021, 1, [(32, 32, 4, 8)] * 3), (2000, 1700, 96, 1, [(128, 128, 8, 1)] * 3), (2001, 1701, 40, 1, [(128, 128, 8, 1)] * 3)])
@pytest.mark.parametrize("tb", [0, 1, 2])
def test_fp32_products_on_the_tiles_they_are_cut_into(eng, m, n, k, batch, cuts, tb):
    """Every tile with and without whole 16-byte pieces and remainders, by what the launch says it was cut into; limit as in `test_fp32_gemm_tiles_and_splits`."""
    rng = np.random.default_rng(m + n + k + tb)
    a = rng.standard_normal((batch, k, m) if tb == 2 else (batch, m, k)).astype(np.float32)
    b = rng.standard_normal((batch, n, k) if tb == 1 else (batch, k, n)).astype(np.float32)
    d = rng.standard_normal((batch, m, n)).astype(np.float32)
    ia, ib, ic, idd = eng.new_tensor(a), eng.new_tensor(b), eng.alloc(d.size + 64), eng.new_tensor(d)
    eng.upload(ic, np.full(d.size + 64, 7.0, np.float32))
    eng.run([op(E.GEMM_EX, a=ia, b=ib, c=ic, d=idd, m=m, n=n, k=k, batch=batch, tb=tb, sa=m * k, sb=k * n, sc=m * n, alpha=0.5, beta=-2.0)])
    assert eng.last_f32_cut() == cuts[tb] and eng.last_variant() == 0x20
    out = eng.download(ic, d.size + 64)
    assert np.all(out[d.size:] == 7.0)
    a64, b64 = a.astype(np.float64), b.astype(np.float64)
    ref = 0.5 * ((a64.transpose(0, 2, 1) if tb == 2 else a64) @ (b64.transpose(0, 2, 1) if tb == 1 else b64)) - 2.0 * d
    assert np.abs(out[:d.size].reshape(ref.shape) - ref).max() <= 10 * 2.0 ** -24 * (k + 4)


def test_fp32_groups_on_64_by_64_tiles(eng):
    """Products of one input, a sum over segments, a SwiGLU pair and its backward, each of 296 tiles of 64 x 64 or more and fewer than 148 of 128 x 128, with remainders; bounds as in the
    tests of those groups."""
    rng = np.random.default_rng(64)
    mk = lambda *sh: rng.standard_normal(sh).astype(np.float32)
    f = lambda v: v.astype(np.float64)
    big = lambda v: np.abs(v).max()
    m, k, ns = 1000, 204, (520, 776, 132)
    x, w = mk(m, k), [mk(k, n) for n in ns]
    ix, iw, ic = put(eng, x, 0), [put(eng, v, 0) for v in w], [eng.alloc(m * n) for n in ns]
    eng.run([op(E.GEMM_GROUP, a=ix, b=iw[0], sa=iw[1], sb=iw[2], c=ic[0], d=ic[1], sc=ic[2], m=m, k=k, n=ns[0], oa=ns[1], ob=ns[2], batch=3, oc=1, tb=0, dt=0)])
    assert eng.last_variant() == 0x29 and eng.last_f32_cut() == (64, 64, 8, 1)
    for g, n in enumerate(ns):
        check(eng.download(ic[g], (m, n)), f(x) @ f(w[g]), False, k)
    n, ks = 1220, (100, 40, 72)
    a, b = [mk(m, q) for q in ks], [mk(n, q) for q in ks]
    ia, ib, io = [put(eng, v, 0) for v in a], [put(eng, v, 0) for v in b], eng.alloc(m * n)
    eng.run([op(E.GEMM_GROUP, c=io, a=ia[0], sa=ia[1], sb=ia[2], b=ib[0], d=ib[1], sc=ib[2], m=m, n=n, k=ks[0], oa=ks[1], ob=ks[2], batch=3, oc=2, tb=1, dt=0)])
    assert eng.last_variant() == 0x29 and eng.last_f32_cut() == (64, 64, 8, 1)
    check(eng.download(io, (m, n)), sum(f(p) @ f(q).T for p, q in zip(a, b)), False, sum(ks))
    for n in (640, 1220):                                # the pair's tiles hold 32 columns of either
        wg, wu = mk(k, n), mk(k, n)
        ig, iu, og, ou, oh = put(eng, wg, 0), put(eng, wu, 0), eng.alloc(m * n), eng.alloc(m * n), eng.alloc(m * n)
        eng.run([op(E.GEMM_GROUP, a=ix, b=ig, sa=iu, c=og, d=ou, sc=oh, m=m, n=n, k=k, batch=2, oc=4, dt=0)])
        assert eng.last_variant() == 0x29 and (n > 640 or eng.last_f32_cut() == (64, 64, 8, 1))
        g, u = f(x) @ f(wg), f(x) @ f(wu)
        s = 1.0 / (1.0 + np.exp(-g))
        check(eng.download(og, (m, n)), g, False, k)
        check(eng.download(ou, (m, n)), u, False, k)
        assert big(eng.download(oh, (m, n)) - g * s * u) <= 4.1 * f32_limit(k) * big(g) * big(u)
    wd, dy = mk(n, k), mk(m, k)
    iwd, idy, idh, idg, idu = put(eng, wd, 0), put(eng, dy, 0), eng.alloc(m * n), eng.alloc(m * n), eng.alloc(m * n)
    eng.run([op(E.GEMM_SB, a=idy, b=iwd, c=idh, m=m, n=n, k=k, batch=1, tb=1, dt=0), op(E.SILU_BWD, a=og, b=ou, d=idh, c=idg, tb=idu, n=m * n, dt=0, oa=1)])
    assert eng.last_variant() == 0x2a and eng.last_f32_cut() == (64, 64, 8, 1)
    dh = f(dy) @ f(wd).T
    assert big(eng.download(idg, (m, n)) - dh * u * s * (1 + g * (1 - s))) <= 2 * f32_limit(k) * big(dh) * big(u) * (2.2 + 0.5 * big(g))
    assert big(eng.download(idu, (m, n)) - dh * g * s) <= 2 * f32_limit(k) * big(dh) * big(g) * 2.1
    assert eng.device_status() == 0


@pytest.mark.parametrize("extra", [0, 1])
@pytest.mark.parametrize("m,n,k", [(256, 256, 64), (520, 392, 320), (1032, 1000, 136), (300, 264, 8)])
def test_swiglu_backward_inside_the_product_that_makes_dh(eng, m, n, k, extra):
    """GEMM_SB (extra 1: GEMM_GROUP mode 2 behind GEMM_XSEG) followed by SILU_BWD with oa = 1 runs as one launch: dg and du against
    float64 — one rounding to bf16 each (2^-8) and the fp32 sum of the product; without oa = 1 two launches that also leave dh."""
    rng = np.random.default_rng(m + n + k + extra)
    r = 16
    mk = lambda *sh: bf(rng.standard_normal(sh).astype(np.float32))
    dY, W, g, u, t, Al = mk(m, k), mk(n, k), bf(3 * mk(m, n)), mk(m, n), mk(m, r), mk(n, r)
    g[0, :8] = [90.0, -90.0, -60.0, 60.0, 0.0, 30.0, -30.0, -126.0]     # saturated gates stay finite
    ins = {nm: put(eng, v, 1) for nm, v in dict(dY=dY, W=W, g=g, u=u, t=t, Al=Al).items()}
    dh64 = dY.astype(np.float64) @ W.T.astype(np.float64) + (t.astype(np.float64) @ Al.T if extra else 0.0)
    sig = 1.0 / (1.0 + np.exp(-g.astype(np.float64)))
    ref = (dh64 * u * sig * (1 + g * (1 - sig)), dh64 * g * sig)
    for fused in (1, 0):
        idh, idg, idu = (eng.alloc(m * n, 2) for _ in range(3))
        prod = [op(E.GEMM_SB, a=ins["dY"], b=ins["W"], c=idh, m=m, n=n, k=k, batch=1, tb=1, dt=1)] if not extra else [
            op(E.GEMM_XSEG, a=ins["t"], sa=ins["Al"], k=r, batch=1),
            op(E.GEMM_GROUP, a=ins["dY"], b=ins["W"], c=idh, m=m, n=n, k=k, batch=1, oc=2, tb=1, dt=1)]
        eng.launch_count(reset=True)
        eng.run(prod + [op(E.SILU_BWD, a=ins["g"], b=ins["u"], d=idh, c=idg, tb=idu, n=m * n, dt=1, oa=fused)])
        assert eng.launch_count() == (1 if fused else 2)
        if fused:
            assert eng.last_variant() == 0x24
        else:
            check(eng.download_bf16(idh, (m, n)), dh64.astype(np.float32), True, k)
        for got, want in zip((eng.download_bf16(idg, (m, n)), eng.download_bf16(idu, (m, n))), ref):
            assert np.isfinite(got).all()
            assert np.abs(got - want).max() <= (2 ** -8 if fused else 2 ** -7) * np.abs(want).max() + 1e-30
    assert eng.device_status() == 0


@pytest.mark.parametrize("r", [8, 32])
@pytest.mark.parametrize("m,n,k", [(256, 256, 64), (520, 392, 320), (1032, 1000, 136)])
def test_swiglu_inside_a_projection_pair_with_adapters(eng, m, n, k, r):
    """GEMM_XSEG + GEMM_GROUP mode 1 + SILU_MUL run as one launch that writes g, u and h = silu(g) * u (one bf16 rounding each)."""
    rng = np.random.default_rng(m + n + k + r)
    mk = lambda *sh: bf(rng.standard_normal(sh).astype(np.float32) * 0.4)
    x, wg, wu, ug, uu, bg, bu = mk(m, k), mk(k, n), mk(k, n), mk(m, r), mk(m, r), mk(r, n), mk(r, n)
    i = [put(eng, v, 1) for v in (x, wg, wu, ug, uu, bg, bu)]
    og, ou, oh = (eng.alloc(m * n, 2) for _ in range(3))
    eng.launch_count(reset=True)
    eng.run([op(E.GEMM_XSEG, a=i[3], b=i[4], sa=i[5], sb=i[6], k=r, batch=2),
             op(E.GEMM_GROUP, a=i[0], b=i[1], sa=i[2], c=og, d=ou, m=m, k=k, n=n, oa=n, batch=2, oc=1, dt=1),
             op(E.SILU_MUL, a=og, b=ou, c=oh, n=m * n, dt=1)])
    assert eng.launch_count() == 1 and eng.last_variant() == (0x28 if m > 1000 else 0x25)      # paired / small-product kernel
    f = lambda v: v.astype(np.float64)
    g, u = f(x) @ f(wg) + f(ug) @ f(bg), f(x) @ f(wu) + f(uu) @ f(bu)
    for o, ref in ((og, g), (ou, u), (oh, g / (1 + np.exp(-g)) * u)):
        got = eng.download_bf16(o, (m, n))
        assert np.abs(got - ref).max() <= 2 ** -8 * np.abs(ref).max()
    assert eng.device_status() == 0


SMALL = [(8, 8, 8), (64, 64, 64), (65, 72, 200), (520, 264, 392), (200, 136, 1024), (129, 1000, 72)]


@pytest.mark.parametrize("tb", [0, 1, 2])
@pytest.mark.parametrize("dt", [1, 2])
@pytest.mark.parametrize("m,n,k", SMALL)
def test_small_products(eng, tb, dt, m, n, k):
    """The small-product kernel at the edges of its 64 x 64 x 64 tiles, with alpha, beta in place and an addend."""
    if tb == 2 and m % 8:
        m += 8 - m % 8
    rng = np.random.default_rng(m + n + k + tb + dt)
    for kw in (dict(), dict(alpha=0.5, beta=1.0), dict(beta=-2.0, addend=True)):
        got, ref = run_gemm(eng, rng, m, n, k, tb, dt, **kw)
        assert eng.last_variant() == 0x26
        check(got, ref, dt == 1, k)


@pytest.mark.parametrize("m,k,ns", [(64, 64, (64, 64, 64)), (200, 136, (128, 64, 72)), (300, 264, (256, 128, 128))])
@pytest.mark.parametrize("rope,r", [(0, 0), (1, 0), (1, 16), (0, 8)])
def test_small_groups_agree_with_the_paired_kernel(eng, m, k, ns, rope, r):
    """Grouped launches (rotary on the first two outputs, low-rank terms, K-segments, SwiGLU both ways) by the small-product kernel and by
    the general ways (paired kernel forced with mask 8; below 256 rows the ops run one by one), each against float64: every arm names
    the kernels that it ran on.  A result of one launch is within one rounding to bf16 (2^-8) of the largest element, one of a
    sequence within three (a product, its low-rank term, the rotation or the activation), the sum of six segments one by one within six."""
    rng = np.random.default_rng(m + k + rope + r)
    val = {}

    def mk(*sh):
        a = bf(rng.standard_normal(sh).astype(np.float32) * 0.3)
        i = put(eng, a, 1)
        val[i] = a.astype(np.float64)
        return i
    T = 40
    ang = np.outer(np.arange(T), 1.0 / 10000 ** (np.arange(32) / 32)).astype(np.float32)
    ic, isn = put(eng, np.cos(ang), 0), put(eng, np.sin(ang), 0)
    x, w, xa, xb = mk(m, k), [mk(k, n) for n in ns], [mk(m, r or 8) for _ in ns], [mk(r or 8, n) for n in ns]
    wt, n1 = [mk(ns[0], k) for _ in ns], ns[0]
    xs = [mk(m, k) for _ in ns]
    xbt, dd = [mk(n1, r or 8) for _ in ns], mk(m, n1)
    g_, u_, w2 = mk(m, n1), mk(m, n1), mk(k, n1)
    rope = rope and ns[0] % 64 == 0
    # float64
    cs, sn = (f(ang.astype(np.float64))[np.arange(m) % T][:, None] for f in (np.cos, np.sin))
    want = []
    for g, n in enumerate(ns):
        y = val[x] @ val[w[g]] + (val[xa[g]] @ val[xb[g]] if r else 0.0)
        if rope and g < 2:
            h = y.reshape(m, n // 64, 64)
            y = np.concatenate([h[..., :32] * cs - h[..., 32:] * sn, h[..., :32] * sn + h[..., 32:] * cs], -1).reshape(m, n)
        want.append(y)
    want.append(sum(val[xs[g]] @ val[wt[g]].T for g in range(3)) + (sum(val[xa[g]] @ val[xbt[g]].T for g in range(3)) + val[dd] if r else 0.0))
    gg = val[x] @ val[w[0]] + (val[xa[0]] @ val[xb[0]] if r else 0.0)
    uu = val[x] @ val[w2] + (val[xa[1]] @ val[xb[0]] if r else 0.0)
    want += [gg, uu, gg / (1 + np.exp(-gg)) * uu]
    dh, sig = val[xs[0]] @ val[wt[0]].T, 1 / (1 + np.exp(-val[g_]))
    want += [dh * val[u_] * sig * (1 + val[g_] * (1 - sig)), dh * val[g_] * sig]

    for mask in (0, 8):
        eng.set_fallback(mask)
        ran = []

        def go(plan):
            eng.launch_count(reset=True)
            eng.run(plan)
            ran.append((eng.launch_count(), eng.last_variant()))
        out = [eng.alloc(m * n, 2) for n in ns] + [eng.alloc(m * n1, 2) for _ in range(7)]
        pre = [op(E.GEMM_XSEG, a=xa[0], b=xa[1], d=xa[2], sa=xb[0], sb=xb[1], sc=xb[2], k=r, batch=3)] if r else []
        go(pre + [op(E.GEMM_GROUP, a=x, b=w[0], sa=w[1], sb=w[2], c=out[0], d=out[1], sc=out[2], m=m, k=k, n=ns[0], oa=ns[1], ob=ns[2],
                     batch=3, oc=1, dt=1, beta=float(ic) if rope else 0.0, gamma=float(isn) if rope else 0.0)])
        pre = [op(E.GEMM_XSEG, a=xa[0], b=xa[1], d=xa[2], sa=xbt[0], sb=xbt[1], sc=xbt[2], k=r, batch=3, c=dd, beta=1.0)] if r else []
        go(pre + [op(E.GEMM_GROUP, c=out[3], a=xs[0], sa=xs[1], sb=xs[2], b=wt[0], d=wt[1], sc=wt[2], m=m, n=n1, k=k, oa=k, ob=k, batch=3,
                     oc=2, tb=1, dt=1)])
        if r:
            go([op(E.GEMM_XSEG, a=xa[0], b=xa[1], sa=xb[0], sb=xb[0], k=r, batch=2),
                op(E.GEMM_GROUP, a=x, b=w[0], sa=w2, c=out[4], d=out[5], m=m, k=k, n=n1, oa=n1, batch=2, oc=1, dt=1),
                op(E.SILU_MUL, a=out[4], b=out[5], c=out[6], n=m * n1, dt=1)])
        else:
            go([op(E.GEMM_GROUP, a=x, b=w[0], sa=w2, c=out[4], d=out[5], sc=out[6], m=m, n=n1, k=k, batch=2, oc=4, dt=1)])
        go([op(E.GEMM_SB, a=xs[0], b=wt[0], c=out[7], m=m, n=n1, k=k, batch=1, tb=1, dt=1),
            op(E.SILU_BWD, a=g_, b=u_, d=out[7], c=out[8], tb=out[9], n=m * n1, dt=1, oa=1)])
        eng.set_fallback(0)
        # a group is one launch; the ops behind it join it from 256 rows and columns on
        if m >= 256:
            assert ran == ([(1, 0x26), (1, 0x26), (1, 0x25 if r else 0x26), (1, 0x24)] if mask == 0 else
                           [(1, 0x23), (1, 0x23), (1, 0x28 if r else 0x23), (1, 0x27)])
        elif mask == 0:
            assert [c for c, _ in ran] == [1, 1, 2 if r else 1, 2] and [v for _, v in ran] == [0x26] * 4
        else:
            assert [c for c, _ in ran] == [3 + (3 if r else 0) + (1 if rope else 0), 6 if r else 3, 5 if r else 3, 2] and 0x26 not in [v for _, v in ran]
        for o, ref, step in zip(out[:7] + out[8:], want, (0, 0, 0, 1, 2, 2, 2, 3, 3)):
            got = eng.download_bf16(o, ref.shape)
            steps = 1 if ran[step][0] == 1 else (6 if step == 1 and r else 3)
            assert np.abs(got - ref).max() <= 1.02 * steps * 2.0 ** -8 * np.abs(ref).max()
    assert eng.device_status() == 0


@pytest.mark.parametrize("tb", [0, 1])
@pytest.mark.parametrize("N,F,R,count", [(1, 768, 8, 1), (33, 776, 16, 1), (70, 3080, 32, 2), (2048, 4096, 16, 1), (2000, 1536, 8, 3), (9600, 768, 16, 1)])
def test_adapter_skinny_products_with_the_depth_split_over_a_cluster(eng, tb, N, F, R, count):
    """LORA_PROJ at token counts that need one, two, four and eight CTAs per token block to fill the GPU, ragged pieces and token
    blocks; the split sums have a fixed order (a second run gives the same bits)."""
    rng = np.random.default_rng(N + F + R + tb)
    X = bf(rng.standard_normal((N, F)).astype(np.float32))
    Ws = [bf(rng.standard_normal((R, F) if tb else (F, R)).astype(np.float32) * 0.1) for _ in range(count)]
    ix, iw = put(eng, X, 1), [put(eng, w, 1) for w in Ws] + [0, 0]
    io = [eng.alloc(N * R + 64, 2) for _ in range(count)] + [0, 0]
    for o_ in io[:count]:
        eng.upload_bf16(o_, np.full(N * R + 64, 3.0, np.float32))
    p = [op(E.LORA_PROJ, a=ix, b=iw[0], d=iw[1], sc=iw[2], c=io[0], oa=io[1], ob=io[2], n=F, k=F, oc=F, m=N, batch=count, tb=tb,
            gamma=float(R), alpha=0.5, dt=1)]
    runs = []
    for _ in range(2):
        eng.run(p)
        assert eng.last_variant() == 0x62
        runs.append([eng.download_bf16(o_, (N * R + 64,)) for o_ in io[:count]])
    for g in range(count):
        assert np.array_equal(runs[0][g], runs[1][g])
        ref = 0.5 * (X.astype(np.float64) @ (Ws[g].T if tb else Ws[g]).astype(np.float64))
        check(runs[0][g][:N * R].reshape(N, R), ref.astype(np.float32), True, F)
        assert np.all(runs[0][g][N * R:] == 3.0)


@pytest.mark.parametrize("tb", [0, 1])
@pytest.mark.parametrize("N,F,R,count,one", [(2031, 1544, 16, 3, 1), (2048, 264, 32, 2, 1), (6401, 136, 32, 3, 1), (1985, 8, 8, 3, 1),
                                             (1984, 1032, 16, 3, 1), (2500, 520, 16, 3, 0), (1200, 4096, 16, 1, 1)])
def test_adapter_skinny_products_of_one_input_as_members(eng, tb, N, F, R, count, one):
    """Products of one X share its stage (from 32 token blocks on, rank * count <= 64, or beyond one wave of CTAs), on both
    sides of that line.  Widths end inside a piece, token counts inside a block; nothing is written past an output."""
    rng = np.random.default_rng(N + F + R + tb)
    Xs = [bf(rng.standard_normal((N, F)).astype(np.float32)) for _ in range(1 if one else count)]
    Xs = Xs * count if one else Xs
    Ws = [bf(rng.standard_normal((R, F) if tb else (F, R)).astype(np.float32) * 0.1) for _ in range(count)]
    ix = [put(eng, X, 1) for X in (Xs[:1] if one else Xs)]
    ix = (ix * count if one else ix) + [0, 0]
    iw = [put(eng, w, 1) for w in Ws] + [0, 0]
    io = [eng.alloc(N * R + 64, 2) for _ in range(count)] + [0, 0]
    for o_ in io[:count]:
        eng.upload_bf16(o_, np.full(N * R + 64, 3.0, np.float32))
    eng.launch_count(reset=True)
    eng.run([op(E.LORA_PROJ, a=ix[0], sa=ix[1], sb=ix[2], b=iw[0], d=iw[1], sc=iw[2], c=io[0], oa=io[1], ob=io[2], n=F, k=F, oc=F,
                m=N, batch=count, tb=tb, gamma=float(R), alpha=0.5, dt=1)])
    assert eng.last_variant() == 0x62 and eng.launch_count() == 1
    for g in range(count):
        got = eng.download_bf16(io[g], (N * R + 64,))
        ref = 0.5 * (Xs[g].astype(np.float64) @ (Ws[g].T if tb else Ws[g]).astype(np.float64))
        assert np.abs(got[:N * R].reshape(N, R) - ref).max() <= 1.02 * 2.0 ** -8 * np.abs(ref).max()      # one rounding to bf16
        assert np.all(got[N * R:] == 3.0)
    assert eng.device_status() == 0


@pytest.mark.parametrize("fused", [0, 1])
def test_a_fused_product_leaves_pending_segments_to_their_group(eng, fused):
    """GEMM_XSEG announces operands for the next GEMM_GROUP; a plain product with its SwiGLU backward may stand between the two,
    run as one launch (oa = 1) or as two."""
    rng = np.random.default_rng(11)
    m, n, k, r = 256, 264, 64, 16
    mk = lambda *sh: bf(rng.standard_normal(sh).astype(np.float32))
    dY, W, g, u, x, w0, w1, xa, xb = mk(m, k), mk(n, k), mk(m, n), mk(m, n), mk(m, k), mk(k, n), mk(k, n), mk(m, r), mk(r, n)
    i = [put(eng, v, 1) for v in (dY, W, g, u, x, w0, w1, xa, xb)]
    idh, idg, idu, o0, o1 = (eng.alloc(m * n, 2) for _ in range(5))
    eng.launch_count(reset=True)
    eng.run([op(E.GEMM_XSEG, a=i[7], b=i[7], sa=i[8], sb=i[8], k=r, batch=2),
             op(E.GEMM_SB, a=i[0], b=i[1], c=idh, m=m, n=n, k=k, batch=1, tb=1, dt=1),
             op(E.SILU_BWD, a=i[2], b=i[3], d=idh, c=idg, tb=idu, n=m * n, dt=1, oa=fused),
             op(E.GEMM_GROUP, a=i[4], b=i[5], sa=i[6], c=o0, d=o1, m=m, k=k, n=n, oa=n, batch=2, oc=1, dt=1)])
    assert eng.launch_count() == 3 - fused
    for o, w in ((o0, w0), (o1, w1)):
        check(eng.download_bf16(o, (m, n)), x.astype(np.float64) @ w.astype(np.float64) + xa.astype(np.float64) @ xb.astype(np.float64), True, k + r)
    assert eng.device_status() == 0


@pytest.mark.parametrize("m,n,k,tb,dt,small", [(1024, 1024, 192, 0, 1, True), (1024, 1024, 200, 0, 1, False), (776, 1024, 192, 1, 1, True),
                                               (776, 1024, 256, 1, 1, False), (1024, 640, 320, 2, 2, True), (1024, 640, 328, 2, 2, False)])
def test_two_waves_of_small_tiles_up_to_the_depth_where_they_pay(eng, m, n, k, tb, dt, small):
    """149 to 296 tiles of 64 x 64: plain products of at most three 64-deep steps, weight gradients of at most five."""
    rng = np.random.default_rng(m + n + k)
    got, ref = run_gemm(eng, rng, m, n, k, tb, dt)
    assert (eng.last_variant() == 0x26) == small
    check(got, ref, dt == 1, k)


# Sizes with more 256-wide tiles than CTA pairs fit the GPU (74), ragged rows and columns: the paired kernel's persistent loop goes round
# with its barriers' phases carried over, and the last row and column tiles are clipped.  Sizes that one wave of 64 x 64 tiles
# covers run on the small-product kernel unless mask 8 asks for the paired one.
def rounding(got, ref):
    """One rounding to bf16 (half an ulp is at most 2^-8 of the element) of an fp32 sum, and 2^-14 of the largest result for that sum: tensor cores
    add k <= 400 products of N(0,1) numbers with at least 23 bits each, an error below k 2^-23 of the largest sum."""
    assert np.isfinite(got).all()
    worst = np.abs(got - ref) - (1.01 * 2.0 ** -8 * np.abs(ref) + 2.0 ** -14 * np.abs(ref).max())
    assert worst.max() <= 0, float(worst.max() / np.abs(ref).max())


def on_paired(mask, small):
    return mask == 8 or not small


WIDE = [(520, 392, 136, True), (1032, 1000, 136, True), (1100, 4360, 72, False)]


@pytest.mark.parametrize("mask", [0, 8])
@pytest.mark.parametrize("extra", [0, 1])
@pytest.mark.parametrize("m,n,k,small", WIDE)
def test_swiglu_backward_on_both_kernels(eng, mask, m, n, k, small, extra):
    rng = np.random.default_rng(m + n + k + extra)
    mk = lambda *sh: bf(rng.standard_normal(sh).astype(np.float32))
    dY, W, g, u, t, Al = mk(m, k), mk(n, k), bf(3 * mk(m, n)), mk(m, n), mk(m, 16), mk(n, 16)
    i = [put(eng, v, 1) for v in (dY, W, g, u, t, Al)]
    idh, idg, idu = (eng.alloc(m * n, 2) for _ in range(3))
    prod = [op(E.GEMM_XSEG, a=i[4], sa=i[5], k=16, batch=1),
            op(E.GEMM_GROUP, a=i[0], b=i[1], c=idh, m=m, n=n, k=k, batch=1, oc=2, tb=1, dt=1)] if extra else [
            op(E.GEMM_SB, a=i[0], b=i[1], c=idh, m=m, n=n, k=k, batch=1, tb=1, dt=1)]
    eng.set_fallback(mask)
    eng.launch_count(reset=True)
    eng.run(prod + [op(E.SILU_BWD, a=i[2], b=i[3], d=idh, c=idg, tb=idu, n=m * n, dt=1, oa=1)])
    eng.set_fallback(0)
    assert eng.launch_count() == 1 and eng.last_variant() == (0x27 if on_paired(mask, small) else 0x24)
    dh = dY.astype(np.float64) @ W.T.astype(np.float64) + (t.astype(np.float64) @ Al.T if extra else 0.0)
    sig = 1.0 / (1.0 + np.exp(-g.astype(np.float64)))
    rounding(eng.download_bf16(idg, (m, n)), dh * u * sig * (1 + g * (1 - sig)))
    rounding(eng.download_bf16(idu, (m, n)), dh * g * sig)
    assert eng.device_status() == 0


@pytest.mark.parametrize("mask", [0, 8])
@pytest.mark.parametrize("r", [0, 16])
@pytest.mark.parametrize("m,n,k,small", [(520, 264, 200, True), (1100, 2056, 200, False)])
def test_swiglu_pair_on_both_kernels(eng, mask, m, n, k, small, r):
    rng = np.random.default_rng(m + n + k + r)
    mk = lambda *sh: bf(rng.standard_normal(sh).astype(np.float32) * 0.4)
    x, wg, wu, ug, uu, bg, bu = mk(m, k), mk(k, n), mk(k, n), mk(m, 16), mk(m, 16), mk(16, n), mk(16, n)
    i = [put(eng, v, 1) for v in (x, wg, wu, ug, uu, bg, bu)]
    og, ou, oh = (eng.alloc(m * n, 2) for _ in range(3))
    plan = [op(E.GEMM_XSEG, a=i[3], b=i[4], sa=i[5], sb=i[6], k=r, batch=2),
            op(E.GEMM_GROUP, a=i[0], b=i[1], sa=i[2], c=og, d=ou, m=m, k=k, n=n, oa=n, batch=2, oc=1, dt=1),
            op(E.SILU_MUL, a=og, b=ou, c=oh, n=m * n, dt=1)] if r else [
            op(E.GEMM_GROUP, a=i[0], b=i[1], sa=i[2], c=og, d=ou, sc=oh, m=m, n=n, k=k, batch=2, oc=4, dt=1)]
    eng.set_fallback(mask)
    eng.launch_count(reset=True)
    eng.run(plan)
    eng.set_fallback(0)
    assert eng.launch_count() == 1
    assert eng.last_variant() == ((0x28 if r else 0x23) if on_paired(mask, small) else (0x25 if r else 0x26))
    f = lambda v: v.astype(np.float64)
    g = f(x) @ f(wg) + (f(ug) @ f(bg) if r else 0.0)
    u = f(x) @ f(wu) + (f(uu) @ f(bu) if r else 0.0)
    for o, ref in ((og, g), (ou, u), (oh, g / (1 + np.exp(-g)) * u)):
        rounding(eng.download_bf16(o, (m, n)), ref)
    assert eng.device_status() == 0


@pytest.mark.parametrize("mask", [0, 8])
@pytest.mark.parametrize("r", [0, 16])
@pytest.mark.parametrize("m,k,ns,small", [(520, 136, (256, 128, 72), True), (2100, 72, (1536, 512, 520), False)])
def test_rotary_projections_on_both_kernels(eng, mask, m, k, ns, small, r):
    """Outputs 0 and 1 leave the launch rotated (rows of several sequences, the last one cut), output 2 does not."""
    rng = np.random.default_rng(m + k + r)
    mk = lambda *sh: bf(rng.standard_normal(sh).astype(np.float32) * 0.4)
    T = 700
    cos, sin = O.rope_tables(T, 64)
    x, w, xa, xb = mk(m, k), [mk(k, n) for n in ns], [mk(m, 16) for _ in ns], [mk(16, n) for n in ns]
    ix, ic, isn = put(eng, x, 1), put(eng, cos, 0), put(eng, sin, 0)
    iw, ia, ib = ([put(eng, v, 1) for v in vs] for vs in (w, xa, xb))
    out = [eng.alloc(m * n, 2) for n in ns]
    pre = [op(E.GEMM_XSEG, a=ia[0], b=ia[1], d=ia[2], sa=ib[0], sb=ib[1], sc=ib[2], k=r, batch=3)] if r else []
    eng.set_fallback(mask)
    eng.launch_count(reset=True)
    eng.run(pre + [op(E.GEMM_GROUP, a=ix, b=iw[0], sa=iw[1], sb=iw[2], c=out[0], d=out[1], sc=out[2], m=m, k=k, n=ns[0], oa=ns[1], ob=ns[2],
                      batch=3, oc=1, dt=1, beta=float(ic), gamma=float(isn))])
    eng.set_fallback(0)
    assert eng.launch_count() == 1 and eng.last_variant() == (0x23 if on_paired(mask, small) else 0x26)
    f = lambda v: v.astype(np.float64)
    c, s = (f(a)[np.arange(m) % T][:, None, :32] for a in (cos.reshape(T, -1), sin.reshape(T, -1)))
    for g, n in enumerate(ns):
        y = f(x) @ f(w[g]) + (f(xa[g]) @ f(xb[g]) if r else 0.0)
        if g < 2:
            h = y.reshape(m, n // 64, 64)
            y = np.concatenate([h[..., :32] * c - h[..., 32:] * s, h[..., :32] * s + h[..., 32:] * c], -1).reshape(m, n)
        rounding(eng.download_bf16(out[g], (m, n)), y)
    assert eng.device_status() == 0


@pytest.mark.parametrize("mask", [0, 8])
@pytest.mark.parametrize("m,n,k,small", [(520, 392, 136, True), (1032, 1000, 136, False), (1100, 4360, 72, False)])
def test_segments_and_addend_on_both_kernels(eng, mask, m, n, k, small):
    rng = np.random.default_rng(m + n + k)
    mk = lambda *sh: bf(rng.standard_normal(sh).astype(np.float32))
    ks = (k, 64, 16)
    A, B, D = [mk(m, q) for q in ks], [mk(n, q) for q in ks], mk(m, n)
    ia, ib = [put(eng, a, 1) for a in A], [put(eng, b, 1) for b in B]
    idd, ic = put(eng, D, 1), eng.alloc(m * n, 2)
    eng.set_fallback(mask)
    eng.launch_count(reset=True)
    eng.run([op(E.GEMM_XSEG, a=ia[2], sa=ib[2], k=ks[2], batch=1, c=idd, beta=-2.0),
             op(E.GEMM_GROUP, c=ic, a=ia[0], sa=ia[1], b=ib[0], d=ib[1], m=m, n=n, k=ks[0], oa=ks[1], batch=2, oc=2, tb=1, dt=1)])
    eng.set_fallback(0)
    assert eng.launch_count() == 1 and eng.last_variant() == (0x23 if on_paired(mask, small) else 0x26)
    rounding(eng.download_bf16(ic, (m, n)), sum(a.astype(np.float64) @ b.T.astype(np.float64) for a, b in zip(A, B)) - 2.0 * D)
    assert eng.device_status() == 0


@pytest.mark.parametrize("mask", [0, 8])
def test_swiglu_of_gates_near_the_end_of_the_fp32_range(eng, mask):
    """silu(g) and its derivative for g around -88, where 1 + exp(-g) lies between 2^126 and 2^128 and the quotient near 1e-37: fused
    launches return it like an IEEE division, to the rounding to bf16 (2^-8) and what the rounding of g log2(e) makes of the exponential
    there (2^-17); beyond, where exp(-g) is infinite, zero is right to 1e-36."""
    m, n, k = 256, 256, 64
    gates = np.array([-88.5, -88.0, -87.5, -87.0, -80.0, -20.0, 20.0, 88.0, -90.0, -120.0, -1e30], np.float32)
    gv = np.resize(gates, n)
    x = np.zeros((m, k), np.float32); x[:, 0] = 1.0
    wg = np.zeros((k, n), np.float32); wg[0] = gv
    wu = np.zeros((k, n), np.float32); wu[0] = 2.0
    i = [put(eng, v, 1) for v in (x, wg, wu)]
    og, ou, oh, idh, idg, idu = (eng.alloc(m * n, 2) for _ in range(6))
    g2, u2 = put(eng, np.tile(gv, (m, 1)), 1), put(eng, np.full((m, n), 2.0, np.float32), 1)
    wt = put(eng, np.concatenate([np.ones((n, 1), np.float32), np.zeros((n, k - 1), np.float32)], 1), 1)
    eng.set_fallback(mask)
    eng.run([op(E.GEMM_GROUP, a=i[0], b=i[1], sa=i[2], c=og, d=ou, sc=oh, m=m, n=n, k=k, batch=2, oc=4, dt=1)])
    assert eng.last_variant() == (0x23 if mask else 0x26)
    eng.run([op(E.GEMM_SB, a=i[0], b=wt, c=idh, m=m, n=n, k=k, batch=1, tb=1, dt=1),
             op(E.SILU_BWD, a=g2, b=u2, d=idh, c=idg, tb=idu, n=m * n, dt=1, oa=1)])
    assert eng.last_variant() == (0x27 if mask else 0x24)
    eng.set_fallback(0)
    g = gv.astype(np.float64)
    with np.errstate(over="ignore"):
        sig = 1 / (1 + np.exp(-g))
    for o, ref in ((oh, 2 * g * sig), (idg, 2 * sig * (1 + g * (1 - sig))), (idu, g * sig)):
        got = eng.download_bf16(o, (m, n))
        assert np.all(np.abs(got - ref) <= np.where(g < -89, 1e-36, (2.0 ** -8 + 2.0 ** -15) * np.abs(ref)))
    assert eng.device_status() == 0


@pytest.mark.parametrize("tb", [0, 1, 2])
@pytest.mark.parametrize("dt,addend", [(1, False), (1, True), (2, False)])
@pytest.mark.parametrize("m,n,k,parts", [(1288, 776, 2064, 2), (1032, 1032, 1352, 2), (520, 776, 1352, 4), (520, 264, 2104, 4), (1544, 1024, 1408, 2)])
def test_tile_depth_shared_over_a_cluster(eng, tb, dt, addend, m, n, k, parts):
    """Few tiles: two or four pairs of CTAs share a tile's depth (uneven parts, ragged last rows, columns and depth; column parts that
    do not exist).  The parts' sums meet in fp32 in a fixed order: the limits of one pair, and the same bits on every run."""
    rng = np.random.default_rng(m + n + k + tb)
    kw = dict(beta=-2.0, addend=True) if addend else dict(alpha=0.5)
    got, ref = run_gemm(eng, rng, m, n, k, tb, dt, fallback=8, **kw)
    assert eng.last_gemm_parts() == parts
    check(got, ref, dt == 1, k)
    again, _ = run_gemm(eng, np.random.default_rng(m + n + k + tb), m, n, k, tb, dt, fallback=8, **kw)
    assert np.array_equal(got, again)
    assert eng.device_status() == 0


@pytest.mark.parametrize("tb", [0, 1, 2])
@pytest.mark.parametrize("m,n,k,parts", [(1288, 776, 2064, 2), (1032, 1032, 1352, 2), (520, 776, 1352, 4), (520, 264, 2104, 4)])
def test_tile_depth_shared_with_a_float_addend(eng, tb, m, n, k, parts):
    """The same with fp32 output and addend: four or two 32-column pieces to a part, which take the staging buffers in turn."""
    test_tile_depth_shared_over_a_cluster(eng, tb, 2, True, m, n, k, parts)


@pytest.mark.parametrize("r", [0, 16])
@pytest.mark.parametrize("m,T,k,ns,parts", [(1032, 258, 1352, (512, 256, 128), 2), (1032, 700, 1352, (512, 128, 264), 2), (520, 260, 1800, (256, 128, 64), 4)])
def test_rotary_projections_of_tiles_shared_over_a_cluster(eng, m, T, k, ns, parts, r):
    """Outputs of whole heads leave the launch rotated, from parts of 128 or 64 columns; the rotation meets the finished sum.
    The sum's 2^-14 in `rounding` holds at this depth, too: errors of 2^-23 in random directions come to sqrt(k) 2^-23, 2^-17.5."""
    rng = np.random.default_rng(m + T + r)
    mk = lambda *sh: bf(rng.standard_normal(sh).astype(np.float32) * 0.4)
    cos, sin = O.rope_tables(T, 64)
    x, w, xa, xb = mk(m, k), [mk(k, n) for n in ns], [mk(m, 16) for _ in ns], [mk(16, n) for n in ns]
    ix, ic, isn = put(eng, x, 1), put(eng, cos, 0), put(eng, sin, 0)
    iw, ia, ib = ([put(eng, v, 1) for v in vs] for vs in (w, xa, xb))
    out = [eng.alloc(m * n, 2) for n in ns]
    pre = [op(E.GEMM_XSEG, a=ia[0], b=ia[1], d=ia[2], sa=ib[0], sb=ib[1], sc=ib[2], k=r, batch=3)] if r else []
    eng.set_fallback(8)
    eng.run(pre + [op(E.GEMM_GROUP, a=ix, b=iw[0], sa=iw[1], sb=iw[2], c=out[0], d=out[1], sc=out[2], m=m, k=k, n=ns[0], oa=ns[1], ob=ns[2],
                      batch=3, oc=1, dt=1, beta=float(ic), gamma=float(isn))])
    eng.set_fallback(0)
    assert (eng.last_variant(), eng.last_gemm_parts()) == (0x23, parts)
    f = lambda v: v.astype(np.float64)
    c, s = (f(a)[np.arange(m) % T][:, None, :32] for a in (cos.reshape(T, -1), sin.reshape(T, -1)))
    for g, n in enumerate(ns):
        y = f(x) @ f(w[g]) + (f(xa[g]) @ f(xb[g]) if r else 0.0)
        if g < 2:
            h = y.reshape(m, n // 64, 64)
            y = np.concatenate([h[..., :32] * c - h[..., 32:] * s, h[..., :32] * s + h[..., 32:] * c], -1).reshape(m, n)
        rounding(eng.download_bf16(out[g], (m, n)), y)
    assert eng.device_status() == 0


@pytest.mark.parametrize("addend", [False, True])
@pytest.mark.parametrize("n,variant,parts", [(776, 0x122, 4), (780, 0x222, 1)])
def test_depth_is_not_shared_for_rows_that_tma_cannot_store(eng, addend, n, variant, parts):
    """Twelve tiles 32 k-blocks deep: four pairs to a tile where rows of C are whole 16-byte pieces, else two parts through the workspace, which
    the cost rule takes only if it knows that the tiles will not be shared."""
    rng = np.random.default_rng(n)
    got, ref = run_gemm(eng, rng, 520, n, 2048, 1, 1, fallback=8, **(dict(beta=-2.0, addend=True) if addend else dict(alpha=0.5)))
    assert (eng.last_variant(), eng.last_gemm_parts()) == (variant, parts)
    check(got, ref, True, 2048)
    assert eng.device_status() == 0


@pytest.mark.parametrize("m,n,k,tb,dt,variant,parts", [
    (512, 2168, 6784, 1, 1, 0x422, 1), (1368, 784, 5264, 2, 1, 0x322, 1), (1472, 744, 7432, 1, 2, 0x422, 1),       # split: more pairs at work
    (1224, 1464, 5240, 1, 1, 0x122, 2), (760, 848, 4464, 1, 1, 0x122, 4)])                                         # shared: no pass over the sums
def test_deep_products_of_few_tiles_are_split_or_shared(eng, m, n, k, tb, dt, variant, parts):
    got, ref = run_gemm(eng, np.random.default_rng(m + n), m, n, k, tb, dt, fallback=8)
    assert (eng.last_variant(), eng.last_gemm_parts()) == (variant, parts)
    check(got, ref, dt == 1, k)
    assert eng.device_status() == 0


@pytest.mark.parametrize("m,k,ns,r,parts", [(1032, 1352, (512, 264, 136), 16, 2), (520, 1800, (264, 136, 72), 8, 4)])
def test_grouped_tiles_shared_over_a_cluster(eng, m, k, ns, r, parts):
    """The same for groups: one input and several outputs with a low-rank term each, and one output summed over K-segments."""
    rng = np.random.default_rng(m + k)
    mk = lambda *sh: bf(rng.standard_normal(sh).astype(np.float32))
    A, Bs, XA, XB = mk(m, k), [mk(k, n) for n in ns], [mk(m, r) for _ in ns], [mk(r, n) for n in ns]
    up = lambda a: put(eng, a, 1)
    ic = [eng.alloc(m * n, 2) for n in ns]
    ia, ib, xa, xb = up(A), [up(b) for b in Bs], [up(a) for a in XA], [up(b) for b in XB]
    eng.set_fallback(8)
    eng.run([op(E.GEMM_XSEG, a=xa[0], b=xa[1], d=xa[2], sa=xb[0], sb=xb[1], sc=xb[2], k=r, batch=3),
             op(E.GEMM_GROUP, a=ia, b=ib[0], sa=ib[1], sb=ib[2], c=ic[0], d=ic[1], sc=ic[2], m=m, k=k, n=ns[0], oa=ns[1], ob=ns[2],
                batch=3, oc=1, dt=1)])
    assert eng.last_gemm_parts() == parts
    for g, n in enumerate(ns):
        check(eng.download_bf16(ic[g], (m, n)), A @ Bs[g] + XA[g] @ XB[g], True, k + r)
    n, ks = 520, (k, 72, 200)
    As, Bt, D = [A, mk(m, 72), mk(m, 200)], [mk(n, q) for q in ks], mk(m, n)
    idd, c = up(D), eng.alloc(m * n, 2)
    ia, ib = [up(a) for a in As], [up(b) for b in Bt]
    eng.run([op(E.GEMM_XSEG, a=0, b=0, d=0, sa=0, sb=0, sc=0, k=0, batch=0, c=idd, beta=1.0),
             op(E.GEMM_GROUP, c=c, a=ia[0], sa=ia[1], sb=ia[2], b=ib[0], d=ib[1], sc=ib[2], m=m, n=n, k=ks[0], oa=ks[1], ob=ks[2], batch=3,
                oc=2, tb=1, dt=1)])
    eng.set_fallback(0)
    assert eng.last_gemm_parts() == 4
    check(eng.download_bf16(c, (m, n)), sum(a @ b.T for a, b in zip(As, Bt)) + D, True, sum(ks))
    assert eng.device_status() == 0


@pytest.mark.parametrize("m,n,k,tb,dt", [(3336, 776, 7816, 0, 1), (3128, 520, 8320, 1, 1), (6408, 264, 4104, 2, 2), (3072, 520, 8512, 2, 2)])
def test_tall_products_walk_their_tiles_in_bands(eng, m, n, k, tb, dt):
    """A above 52 MB: bands of twelve row tiles, the last one of two, one, two and twelve; every tile of the output is written once."""
    assert 2 * m * k > 52000000
    got, ref = run_gemm(eng, np.random.default_rng(m + n), m, n, k, tb, dt, fallback=8)
    check(got, ref, dt == 1, k)
    assert eng.device_status() == 0


F32_GROUPS = [(5, 7, (3, 9, 2)), (33, 66, (40, 8, 1)),              # rows that are no whole 16-byte pieces, less than a tile
              (512, 256, (256, 128, 128)), (100, 1100, (36, 4, 200)),    # 64 x 32 and 32 x 32 tiles, the depth over a cluster
              (700, 72, (520, 264, 132)), (1300, 36, (1032, 776, 516))]  # 32 x 32, 64 x 64 and 128 x 128 tiles


def f32_limit(k):
    return 3e-6 * max(1.0, np.sqrt(k) / 4)             # as in `check`, of the largest element


@pytest.mark.parametrize("tb", [0, 1, 2])
@pytest.mark.parametrize("m,k,ns", F32_GROUPS)
def test_fp32_products_of_one_input_as_one_launch(eng, tb, m, k, ns):
    rng = np.random.default_rng(m + k + tb)
    mk = lambda *sh: rng.standard_normal(sh).astype(np.float32)
    x, w = mk(*((k, m) if tb == 2 else (m, k))), [mk(*((n, k) if tb == 1 else (k, n))) for n in ns]
    ix, iw, ic = put(eng, x, 0), [put(eng, v, 0) for v in w], [put(eng, np.full((m, n), np.nan, np.float32), 0) for n in ns]
    eng.launch_count(reset=True)
    eng.run([op(E.GEMM_GROUP, a=ix, b=iw[0], sa=iw[1], sb=iw[2], c=ic[0], d=ic[1], sc=ic[2], m=m, k=k, n=ns[0], oa=ns[1], ob=ns[2], batch=3, oc=1, tb=tb, dt=0)])
    assert (eng.launch_count(), eng.last_variant()) == (1, 0x29)
    f = lambda v, t: (v.T if t else v).astype(np.float64)
    for g, n in enumerate(ns):
        check(eng.download(ic[g], (m, n)), f(x, tb == 2) @ f(w[g], tb == 1), False, k)
    # an output that another member reads: the members run one by one, the last product meets the first one's result
    if tb == 0 and ns[0] * m >= k * ns[2]:
        eng.run([op(E.GEMM_GROUP, a=ix, b=iw[0], sa=iw[1], sb=ic[0], c=ic[0], d=ic[1], sc=ic[2], m=m, k=k, n=ns[0], oa=ns[1], ob=ns[2], batch=3, oc=1, dt=0)])
        assert eng.last_variant() == 0x20
        first = eng.download(ic[0], (m * ns[0],))[:k * ns[2]].reshape(k, ns[2])
        check(eng.download(ic[2], (m, ns[2])), f(x, 0) @ f(first, 0), False, k)


@pytest.mark.parametrize("addend", [0, 1, 2])                       # none, one of its own, the output itself
@pytest.mark.parametrize("m,k,ns", F32_GROUPS)
def test_fp32_sum_over_segments_as_one_launch(eng, m, k, ns, addend):
    rng = np.random.default_rng(m + k + addend)
    mk = lambda *sh: rng.standard_normal(sh).astype(np.float32)
    n, r, ks = ns[0], 4, (k,) + ns[1:]
    a, b, xa, xb, d = [mk(m, q) for q in ks], [mk(n, q) for q in ks], mk(m, r), mk(n, r), mk(m, n)
    ia, ib, ixa, ixb, idd = [put(eng, v, 0) for v in a], [put(eng, v, 0) for v in b], put(eng, xa, 0), put(eng, xb, 0), put(eng, d, 0)
    ic = idd if addend == 2 else put(eng, np.full((m, n), np.nan, np.float32), 0)
    eng.launch_count(reset=True)
    eng.run([op(E.GEMM_XSEG, a=ixa, sa=ixb, k=r, batch=1, c=idd if addend else 0, beta=-2.0),
             op(E.GEMM_GROUP, c=ic, a=ia[0], sa=ia[1], sb=ia[2], b=ib[0], d=ib[1], sc=ib[2], m=m, n=n, k=ks[0], oa=ks[1], ob=ks[2], batch=3, oc=2, tb=1, dt=0,
                alpha=0.5)])
    assert (eng.launch_count(), eng.last_variant()) == (1, 0x29)
    f = lambda v: v.astype(np.float64)
    ref = 0.5 * (sum(f(x) @ f(w).T for x, w in zip(a, b)) + f(xa) @ f(xb).T) - (2.0 * f(d) if addend else 0.0)
    check(eng.download(ic, (m, n)), ref, False, sum(ks) + r)


@pytest.mark.parametrize("m,k,ns", F32_GROUPS)
def test_fp32_swiglu_pair_and_its_backward_inside_their_products(eng, m, k, ns):
    """g, u and h = silu(g) u from one launch; dg and du from the product that makes dh, which is not written.  Bounds: the error of a product, `f32_limit` of its
    largest element, times what the outputs' derivatives make of it (silu' and sigmoid' g up to 1.1 and 0.5, sigmoid up to 1), and as much again for their own arithmetic."""
    rng = np.random.default_rng(m + k)
    mk = lambda *sh: rng.standard_normal(sh).astype(np.float32)
    n = ns[0]
    x, wg, wu = mk(m, k), mk(k, n), mk(k, n)
    ix, ig, iu = put(eng, x, 0), put(eng, wg, 0), put(eng, wu, 0)
    og, ou, oh = (put(eng, np.full((m, n), np.nan, np.float32), 0) for _ in range(3))
    eng.launch_count(reset=True)
    eng.run([op(E.GEMM_GROUP, a=ix, b=ig, sa=iu, c=og, d=ou, sc=oh, m=m, n=n, k=k, batch=2, oc=4, dt=0)])
    assert (eng.launch_count(), eng.last_variant()) == (1, 0x29)
    f = lambda v: v.astype(np.float64)
    big = lambda v: np.abs(v).max()
    g, u = f(x) @ f(wg), f(x) @ f(wu)
    sig = lambda v: 1.0 / (1.0 + np.exp(-v))
    check(eng.download(og, (m, n)), g, False, k)
    check(eng.download(ou, (m, n)), u, False, k)
    assert big(eng.download(oh, (m, n)) - g * sig(g) * u) <= 2 * f32_limit(k) * (1.1 * big(u) * big(g) + big(g) * big(u))
    dy, wd = mk(m, k), mk(n, k)
    idy, iwd, idh, idg, idu = put(eng, dy, 0), put(eng, wd, 0), put(eng, np.full((m, n), 7.0, np.float32), 0), eng.alloc(m * n), eng.alloc(m * n)
    eng.launch_count(reset=True)
    eng.run([op(E.GEMM_SB, a=idy, b=iwd, c=idh, m=m, n=n, k=k, batch=1, tb=1, dt=0), op(E.SILU_BWD, a=og, b=ou, d=idh, c=idg, tb=idu, n=m * n, dt=0, oa=1)])
    assert (eng.launch_count(), eng.last_variant()) == (1, 0x2a) and np.all(eng.download(idh, (m, n)) == 7.0)
    dh, s = f(dy) @ f(wd).T, sig(g)
    assert big(eng.download(idg, (m, n)) - dh * u * s * (1 + g * (1 - s))) <= 2 * f32_limit(k) * big(dh) * big(u) * (1.1 + 0.5 * big(g) + 1.1)
    assert big(eng.download(idu, (m, n)) - dh * g * s) <= 2 * f32_limit(k) * big(dh) * big(g) * (1 + 1.1)
    # without the mark the gradient of h is kept: two launches
    eng.run([op(E.GEMM_SB, a=idy, b=iwd, c=idh, m=m, n=n, k=k, batch=1, tb=1, dt=0), op(E.SILU_BWD, a=og, b=ou, d=idh, c=idg, tb=idu, n=m * n, dt=0)])
    check(eng.download(idh, (m, n)), dh, False, k)


@pytest.mark.parametrize("tb", [0, 2])
@pytest.mark.parametrize("dt,m,n,k", [(1, 320, 448, 200), (2, 256, 256, 64), (1, 576, 1088, 72), (1, 320, 456, 200), (2, 328, 448, 200)])
def test_operands_of_whole_64_blocks_and_others(eng, tb, dt, m, n, k):
    """M- and N-major operands travel as two blocks of 64 columns in one instruction where their rows are whole blocks, ending in the first or the
    second of a pair, else one by one."""
    got, ref = run_gemm(eng, np.random.default_rng(m + n + k), m, n, k, tb, dt, fallback=8)
    check(got, ref, dt == 1, k)
    assert eng.device_status() == 0


@pytest.mark.parametrize("tb", [0, 1, 2])
@pytest.mark.parametrize("dt,addend", [(1, False), (1, True), (2, False), (2, True)])
@pytest.mark.parametrize("m,n,k,width", [(2000, 1504, 640, 192), (2000, 1416, 712, 192), (1304, 776, 1000, 128), (1288, 640, 1000, 128)])
def test_narrow_tiles_where_wide_ones_leave_pairs_idle(eng, tb, dt, addend, m, n, k, width):
    """Tiles of 192 and 128 columns: last tiles of 160, 72, 8 and 128 columns, rows of B that are whole blocks of 32 or 64 and rows that are not.  A column's sum
    does not depend on the tile: where the wide ones share no depth (40 or more of them) the bits are theirs."""
    kw = dict(beta=-2.0, addend=True) if addend else dict(alpha=0.5)
    got, ref = run_gemm(eng, np.random.default_rng(m + n), m, n, k, tb, dt, **kw)
    assert (eng.last_variant(), eng.last_gemm_parts(), eng.last_gemm_width()) == (0x122, 1, width)
    check(got, ref, dt == 1, k)
    wide, _ = run_gemm(eng, np.random.default_rng(m + n), m, n, k, tb, dt, fallback=8, **kw)
    assert eng.last_gemm_width() == 256 and (width != 192 or np.array_equal(got, wide))
    assert eng.device_status() == 0


@pytest.mark.parametrize("m,n,k,tb,dt,width,split", [
    (2520, 2920, 104, 1, 1, 256, 1), (5720, 816, 128, 2, 1, 192, 1), (2176, 3456, 128, 0, 2, 256, 1), (1544, 2176, 568, 2, 2, 256, 1), (4200, 728, 128, 2, 1, 192, 1),
    (768, 2816, 256, 2, 1, 128, 1), (280, 1888, 3792, 2, 1, 256, 3)])
def test_wide_tiles_where_the_epilogue_is_the_round(eng, m, n, k, tb, dt, width, split):
    """A product of few k-blocks pays an epilogue for each round of tiles, so that more rounds of narrow tiles are no gain; one of many k-blocks is split over the
    workspace rather than run on tiles of 128 columns whose k-blocks take as long as they do."""
    got, ref = run_gemm(eng, np.random.default_rng(m + n), m, n, k, tb, dt)
    assert (eng.last_variant(), eng.last_gemm_width()) == (0x22 + 0x100 * split, width)
    check(got, ref, dt == 1, k)
    assert eng.device_status() == 0


@pytest.mark.parametrize("mode,m,dims,depth,tb,parts", [(2, 1072, (232, 2456), 312, 1, 4), (2, 264, (40, 1864, 184), 664, 1, 4), (1, 1528, (40, 168, 288), 3304, 0, 2), (1, 408, (136, 1312), 2696, 1, 4)])
def test_wide_tiles_where_rows_do_not_start_on_32_bytes(eng, mode, m, dims, depth, tb, parts):
    """Sums over segments (dims their depths, depth the columns) and outputs of one input (dims their columns): k-blocks of narrow tiles take longer there than the shared depth of wide ones."""
    rng = np.random.default_rng(m)
    mk = lambda *sh: bf(rng.standard_normal(sh, dtype=np.float32))
    n, k = (depth, dims[0]) if mode == 2 else (dims[0], depth)
    a = [mk(m, d) for d in dims] if mode == 2 else [mk(m, k)]
    b = [mk(n, d) if mode == 2 else mk(d, k) if tb == 1 else mk(k, d) for d in dims]
    ia, ib = [put(eng, v, 1) for v in a] + [0, 0], [put(eng, v, 1) for v in b] + [0]
    ic = [eng.alloc(m * (n if mode == 2 else d), 2) for d in dims] + [0]
    oa, ob = dims[1], dims[2] if len(dims) > 2 else 0
    if mode == 2:
        eng.run([op(E.GEMM_GROUP, c=ic[0], a=ia[0], sa=ia[1], sb=ia[2], b=ib[0], d=ib[1], sc=ib[2], m=m, n=n, k=k, oa=oa, ob=ob, batch=len(dims), oc=2, tb=1, dt=1)])
        got = [(ic[0], n, sum(p.astype(np.float64) @ q.T for p, q in zip(a, b)), sum(dims))]
    else:
        eng.run([op(E.GEMM_GROUP, a=ia[0], b=ib[0], sa=ib[1], sb=ib[2], c=ic[0], d=ic[1], sc=ic[2], m=m, n=n, k=k, oa=oa, ob=ob, batch=len(dims), oc=1, tb=tb, dt=1)])
        got = [(i, d, a[0].astype(np.float64) @ (q.T if tb == 1 else q), k) for i, d, q in zip(ic, dims, b)]
    assert (eng.last_variant(), eng.last_gemm_width(), eng.last_gemm_parts()) == (0x23, 256, parts)
    for i, w, ref, terms in got:
        check(eng.download_bf16(i, (m, w)), ref, True, terms)
    assert eng.device_status() == 0


@pytest.mark.parametrize("m,n,k,tb,parts", [(1040, 720, 2016, 0, 4), (1040, 720, 2016, 2, 4), (2440, 696, 1880, 1, 2), (2248, 584, 3496, 2, 2)])
def test_fp32_outputs_keep_the_partial_sums_of_a_shared_depth(eng, m, n, k, tb, parts):
    """The tensor core's accumulator loses with each step, so that one chain over the depth errs by as many times more as there are parts (2.1 and 4.4 times on one B200).  The default
    route against the forced paired kernel, which shares these depths; a bound of 1.5 lies between no part lost and two made one.  Alone, and as a group of two outputs."""
    rng = np.random.default_rng(m + k)
    a, b = bf(rng.standard_normal((k, m) if tb == 2 else (m, k), dtype=np.float32)), bf(rng.standard_normal((n, k) if tb == 1 else (k, n), dtype=np.float32))
    ref = (a.T if tb == 2 else a).astype(np.float64) @ (b.T if tb == 1 else b)
    ia, ib, ic, idd = put(eng, a, 1), put(eng, b, 1), eng.alloc(m * n), eng.alloc(m * n)
    alone = [op(E.GEMM_SB, a=ia, b=ib, c=ic, m=m, n=n, k=k, batch=1, tb=tb, dt=2)]
    half = 256                                           # the group: columns of the same product, in as many tiles
    hb = [np.ascontiguousarray(v) for v in ((b[:half], b[half:]) if tb == 1 else (b[:, :half], b[:, half:]))]
    ih = [put(eng, v, 1) for v in hb]
    group = [op(E.GEMM_GROUP, a=ia, b=ih[0], sa=ih[1], c=ic, d=idd, m=m, k=k, n=half, oa=n - half, batch=2, oc=1, tb=tb, dt=2)]
    for plan in (alone, group):
        errs = []
        for mask in (0, 8):
            eng.set_fallback(mask)
            eng.run(plan)
            eng.set_fallback(0)
            errs.append(np.linalg.norm(eng.download(ic, (m, n) if plan is alone else (m, half)) - (ref if plan is alone else ref[:, :half])))
            assert (eng.last_gemm_width(), eng.last_gemm_parts()) == (256, parts)
        assert errs[0] <= 1.5 * errs[1], errs
    assert eng.device_status() == 0


@pytest.mark.parametrize("dt", [1, 2])
@pytest.mark.parametrize("m,n,k,width", [(2000, 1501, 640, 192), (2000, 1411, 712, 192), (1304, 777, 1000, 128), (1288, 642, 1000, 128)])
def test_narrow_tiles_whose_rows_are_no_whole_pieces(eng, dt, m, n, k, width):
    """A B^T with any n: the threads of the epilogue store (and read the addend), the last tile holding 157, 67, 9 and 2 columns."""
    for kw in (dict(alpha=0.5), dict(beta=-2.0, addend=True)):
        got, ref = run_gemm(eng, np.random.default_rng(m + n), m, n, k, 1, dt, **kw)
        assert (eng.last_variant(), eng.last_gemm_parts(), eng.last_gemm_width()) == (0x122, 1, width)
        check(got, ref, dt == 1, k)
    assert eng.device_status() == 0


def test_tall_groups_walk_their_tiles_in_bands(eng):
    """A above 52 MB as in `test_tall_products_walk_their_tiles_in_bands`, in groups: several outputs of one input, a sum whose segments are above it together, a SwiGLU pair."""
    rng = np.random.default_rng(52)
    mk = lambda *sh: bf(rng.standard_normal(sh, dtype=np.float32))
    m, k, ns = 3336, 7816, (264, 136, 72)
    assert 2 * m * k > 52000000
    x, ws = mk(m, k), [mk(k, n) for n in ns]
    ix, iw, ic = put(eng, x, 1), [put(eng, w, 1) for w in ws], [eng.alloc(m * n, 2) for n in ns]
    eng.run([op(E.GEMM_GROUP, a=ix, b=iw[0], sa=iw[1], sb=iw[2], c=ic[0], d=ic[1], sc=ic[2], m=m, k=k, n=ns[0], oa=ns[1], ob=ns[2], batch=3, oc=1, tb=0, dt=1)])
    assert eng.last_variant() == 0x23
    for n, w, c in zip(ns, ws, ic):
        check(eng.download_bf16(c, (m, n)), x @ w, True, k)
    g, u = x @ ws[0], x @ (wu := mk(k, ns[0]))
    og, ou, oh = (eng.alloc(m * ns[0], 2) for _ in range(3))
    eng.run([op(E.GEMM_GROUP, a=ix, b=iw[0], sa=put(eng, wu, 1), c=og, d=ou, sc=oh, m=m, n=ns[0], k=k, batch=2, oc=4, dt=1)])
    assert eng.last_variant() == 0x23
    for o, ref in ((og, g), (ou, u), (oh, g / (1 + np.exp(-np.clip(g, -80, None))) * u)):
        check(eng.download_bf16(o, (m, ns[0])), ref, True, k)
    ks, n = (3904, 2600, 1352), 520
    assert 2 * m * sum(ks) > 52000000
    a, b = [mk(m, q) for q in ks], [mk(n, q) for q in ks]
    ia, ib, io = [put(eng, v, 1) for v in a], [put(eng, v, 1) for v in b], eng.alloc(m * n, 2)
    eng.run([op(E.GEMM_GROUP, c=io, a=ia[0], sa=ia[1], sb=ia[2], b=ib[0], d=ib[1], sc=ib[2], m=m, n=n, k=ks[0], oa=ks[1], ob=ks[2], batch=3, oc=2, tb=1, dt=1)])
    assert eng.last_variant() == 0x23
    check(eng.download_bf16(io, (m, n)), sum(p @ q.T for p, q in zip(a, b)), True, sum(ks))
    assert eng.device_status() == 0


@pytest.mark.parametrize("r", [0, 16])
@pytest.mark.parametrize("m,k,ns,width", [(3000, 640, (768, 192, 192), 192), (2904, 264, (704, 192, 128), 192), (1800, 72, (576, 64, 72), 128)])
def test_narrow_tiles_of_groups_have_the_bits_of_wide_ones(eng, m, k, ns, width, r):
    """Projections of one input, two of them rotated, with and without low-rank terms; sums over segments with an addend; the SwiGLU backward.  Against the wide
    tiles of the forced kernel (too many to share their depth, which has another order), whose tests compare them with float64."""
    rng = np.random.default_rng(m + k + r)
    mk = lambda *sh: put(eng, bf(rng.standard_normal(sh).astype(np.float32) * 0.3), 1)
    cos, sin = O.rope_tables(m // 4, 64)
    ix, iw, ia, ib = mk(m, k), [mk(k, n) for n in ns], [mk(m, 16) for _ in ns], [mk(16, n) for n in ns]
    ic, isn = put(eng, cos, 0), put(eng, sin, 0)
    n, gs, wt = ns[0], [mk(m, q) for q in ns], [mk(ns[0], q) for q in ns]
    res, g, u = mk(m, n), mk(m, n), mk(m, n)
    outs = [eng.alloc(m * q, 2) for q in ns] + [eng.alloc(m * n, 2) for _ in range(4)]
    xseg = [op(E.GEMM_XSEG, a=ia[0], b=ia[1], d=ia[2], sa=ib[0], sb=ib[1], sc=ib[2], k=r, batch=3)] if r else []
    addend = [op(E.GEMM_XSEG, a=0, b=0, d=0, sa=0, sb=0, sc=0, k=0, batch=0, c=res, beta=1.0)] if r else []
    q, kk, v, y, dh, dg, du = outs
    plans = [xseg + [op(E.GEMM_GROUP, a=ix, b=iw[0], sa=iw[1], sb=iw[2], c=q, d=kk, sc=v, m=m, k=k, n=ns[0], oa=ns[1], ob=ns[2], batch=3, oc=1, dt=1,
                        beta=float(ic), gamma=float(isn))],
             addend + [op(E.GEMM_GROUP, c=y, a=gs[0], sa=gs[1], sb=gs[2], b=wt[0], d=wt[1], sc=wt[2], m=m, n=n, k=ns[0], oa=ns[1], ob=ns[2], batch=3, oc=2, tb=1, dt=1)],
             [op(E.GEMM_SB, a=gs[0], b=wt[0], c=dh, m=m, n=n, k=ns[0], batch=1, tb=1, dt=1), op(E.SILU_BWD, a=g, b=u, d=dh, c=dg, tb=du, n=m * n, dt=1, oa=1)]]
    runs, widths = [], []
    for mask in (0, 8):
        eng.set_fallback(mask)
        for p in plans:
            eng.run(p)
            widths.append(eng.last_gemm_width())
        eng.set_fallback(0)
        runs.append([eng.download_bf16(o, (m, w)) for o, w in zip(outs, list(ns) + [n, n, n, n]) if o != dh])
    assert widths[0] == width and 256 not in widths[:3] and widths[3:] == [256] * 3
    for a, b in zip(*runs):
        assert np.array_equal(a, b)
    assert eng.device_status() == 0


def test_narrow_tiles_only_while_nothing_runs_beside_the_chain(eng):
    """Products on the side stream take the pairs that wide tiles leave idle: behind the first switch of a plan to another stream the tiles are wide, and a new plan starts over."""
    rng = np.random.default_rng(3)
    mk = lambda *sh: put(eng, bf(rng.standard_normal(sh).astype(np.float32)), 1)
    m, n, k = 2000, 1504, 640
    a, b, c, d = mk(m, k), mk(k, n), eng.alloc(m * n, 2), eng.alloc(m * n, 2)
    prod = lambda out: [op(E.GEMM_SB, a=a, b=b, c=out, m=m, n=n, k=k, batch=1, dt=1)]
    eng.run(prod(c))
    assert eng.last_gemm_width() == 192
    eng.run([op(E.EVENT, tb=1, sa=0, oa=1), op(E.EVENT, tb=2, sa=2, oa=1), op(E.STREAM, tb=2)] + prod(d) + [op(E.EVENT, tb=1, sa=2, oa=2), op(E.STREAM, tb=0)] + prod(c) +
            [op(E.EVENT, tb=2, sa=0, oa=2)])
    assert eng.last_gemm_width() == 256
    assert np.array_equal(eng.download_bf16(c, (m, n)), eng.download_bf16(d, (m, n)))
    eng.run(prod(c))
    assert eng.last_gemm_width() == 192
