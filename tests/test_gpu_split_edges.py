"""GPU: sizes at which a kernel changes how it splits its work (slice, tile and list limits), against the fp64 oracle."""
import numpy as np
import pytest
import torch

from conftest import seeded_qkv

pytestmark = pytest.mark.gpu

# stored results: a few units in the last place of the 16-bit format for |O| <~ 4; fp32: sums of fp32 products
TOL = {torch.float32: 1e-5, torch.float16: 2e-3, torch.bfloat16: 1.6e-2}


@pytest.fixture()
def capi(pkg):
    c = pkg.capi
    c.set_path(c.PATH_AUTO)
    yield c
    c.set_path(c.PATH_AUTO)
    assert c.last_device_error() == 0


def dev(x):
    return torch.from_numpy(np.ascontiguousarray(x)).cuda()


def state(n, d, dtype):
    return (torch.full((n,), float("-inf"), device="cuda", dtype=dtype), torch.zeros(n, device="cuda", dtype=dtype),
            torch.zeros(n, d, device="cuda", dtype=dtype))


def close(st, want, tol, what):
    m, l, O = (t.double().cpu().numpy() for t in st)
    assert np.array_equal(np.isnan(O), np.isnan(want[2])), what
    assert np.nanmax(np.abs(O - want[2])) <= tol, f"{what}: O {np.nanmax(np.abs(O - want[2])):.3e}"
    fin = np.isfinite(want[0])
    assert np.array_equal(np.isfinite(m), fin), what
    np.testing.assert_allclose(m[fin], want[0][fin], rtol=4 * tol, atol=4 * tol, err_msg=what)
    np.testing.assert_allclose(l, want[1], rtol=4 * tol, atol=1e-6, err_msg=what)


def csr_of_lengths(lengths, Lk, seed):
    """Distinct ascending random columns, `lengths[r]` of them in row r."""
    rng = np.random.default_rng(seed)
    off = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int64)
    col = np.concatenate([np.sort(rng.choice(Lk, n, replace=False)) for n in lengths] + [[]]).astype(np.int32)
    return off, col


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("d", [32, 64, 128])
def test_16bit_rows_around_the_slice_length(capi, orc, dtype, d):
    """Rows of one slice exactly, one entry more, several slices with a remainder, an empty row; CSR and COO."""
    Lk = 5000
    lengths = [0, 1, 255, 256, 257, 512, 513, 4999, 31, 33, 2048, 0, 300] + [7] * 50 + [1025]
    off, col = csr_of_lengths(lengths, Lk, d)
    n = len(lengths)
    Q, K, V = seeded_qkv(n, d, 11 + d, Lk=Lk)
    q, k, v = (dev(x).to(dtype) for x in (Q, K, V))
    Qr, Kr, Vr = (x.float().cpu().numpy() for x in (q, k, v))
    want = orc.csr_forward(Qr, Kr, Vr, off, col, use_nan=True)
    st = state(n, d, dtype)
    capi.forward_16("csr", q, k, v, *st, row_off=dev(off), col_ind=dev(col), use_nan=True)
    close(st, want, TOL[dtype], f"csr {dtype} d={d}")
    rows = np.repeat(np.arange(n), lengths).astype(np.int64)
    st = state(n, d, dtype)
    capi.forward_16("coo", q, k, v, *st, row_ind=dev(rows), col_ind=dev(col), use_nan=True)
    close(st, want, TOL[dtype], f"coo {dtype} d={d}")


@pytest.mark.parametrize("d", [32, 64, 128])
@pytest.mark.parametrize("Lk,launches", [(300, 1), (1024, 1), (1025, 2)])
def test_16bit_short_masks_need_no_slice_list(capi, orc, d, Lk, launches):
    """Up to 1024 keys the four warps of a CTA share a long row and nothing is listed: one launch."""
    lengths = [0, 1, min(Lk, 255), min(Lk, 256), min(Lk, 257), Lk, Lk, Lk, Lk, 31, 0, min(Lk, 513)] * 3
    off, col = csr_of_lengths(lengths, Lk, d)
    n = len(lengths)
    q, k, v = (dev(x).half() for x in seeded_qkv(n, d, 17 + d, Lk=Lk))
    want = orc.csr_forward(*(x.float().cpu().numpy() for x in (q, k, v)), off, col, use_nan=True)
    st, off, col = state(n, d, torch.float16), dev(off), dev(col)
    before = capi.launch_count()
    capi.forward_16("csr", q, k, v, *st, row_off=off, col_ind=col, use_nan=True)
    assert capi.launch_count() - before == launches
    close(st, want, TOL[torch.float16], f"Lk={Lk} d={d}")


@pytest.mark.parametrize("kind", ["csr", "coo"])
@pytest.mark.parametrize("n,dtype", [(3000, torch.float16), (5000, torch.bfloat16), (70001, torch.float16)])
def test_16bit_slice_list_among_the_rows(capi, orc, kind, n, dtype):
    """The list blocks follow the first 888 blocks of rows: behind all of them (3000 rows), among them (5000), with CTAs that claim
    eight rows (70001); long rows on both sides of the list. Twice on one state: m and O stay, l doubles."""
    Lk, d = 3000, 64
    lengths = [(3, 1, 0, 7)[r % 4] for r in range(n)]
    for r in (0, 1, 2, n // 3, 2900, n - 2, n - 1):
        lengths[r] = 257 + (r * 37) % 2500
    off, col = csr_of_lengths(lengths, Lk, n)
    q, k, v = (dev(x).to(dtype) for x in seeded_qkv(n, d, n % 100, Lk=Lk))
    m, l, O = orc.csr_forward(*(x.float().cpu().numpy() for x in (q, k, v)), off, col)
    kw = (dict(row_off=dev(off)) if kind == "csr" else dict(row_ind=dev(np.repeat(np.arange(n), lengths).astype(np.int64))))
    st = state(n, d, dtype)
    for times in (1, 2):
        capi.forward_16(kind, q, k, v, *st, col_ind=dev(col), **kw)
        close(st, (m, times * l, O), times * TOL[dtype], f"{kind} n={n} call {times}")


def test_16bit_longer_slices_of_a_huge_mask(capi, orc):
    """From 33 million entries on slices are longer (512 slots for 2^26), so that the scratch stays bounded. Only the first
    entries of the column array belong to rows here."""
    Lk, d, nnz = 5000, 64, 1 << 26
    lengths = [300, 511, 512, 513, 1024, 1025, 4999, 0, 5] * 3
    off, col = csr_of_lengths(lengths, Lk, 1)
    n = len(lengths)
    q, k, v = (dev(x).half() for x in seeded_qkv(n, d, 8, Lk=Lk))
    want = orc.csr_forward(*(x.float().cpu().numpy() for x in (q, k, v)), off, col)
    cols = torch.zeros(nnz, dtype=torch.int32, device="cuda")
    cols[:len(col)] = dev(col)
    st = state(n, d, torch.float16)
    capi.forward_16("csr", q, k, v, *st, row_off=dev(off), col_ind=cols)
    close(st, want, TOL[torch.float16], "longer slices")


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("d", [32, 64, 128])
def test_16bit_more_slices_than_the_list_holds(capi, orc, dtype, d):
    """The slice list is sized from nnz. Rows that share their entries (offsets that fall back, all of them inside the column
    array) and an nnz below the last offset need more room: every long row is walked all the same."""
    Lk, n = 5000, 1300
    shared = np.sort(np.random.default_rng(d).choice(Lk, n, replace=False)).astype(np.int32)
    pairs = 70  # rows 0, 2, 4, ... hold [0, n); the rows between them end before they begin and are empty
    off = np.array([0, n] * pairs + [0], dtype=np.int64)
    valid = np.concatenate([[0], np.cumsum([n, 0] * pairs)]).astype(np.int64)
    q, k, v = (dev(x).to(dtype) for x in seeded_qkv(2 * pairs, d, 21 + d, Lk=Lk))
    Qr, Kr, Vr = (x.float().cpu().numpy() for x in (q, k, v))
    st = state(2 * pairs, d, dtype)
    capi.forward_16("csr", q, k, v, *st, row_off=dev(off), col_ind=dev(shared), use_nan=True)
    close(st, orc.csr_forward(Qr, Kr, Vr, valid, np.tile(shared, pairs), use_nan=True), TOL[dtype], f"shared {dtype} d={d}")
    lengths = [300, 7, 256, 0, 4999, 257, 1, 700] * 12
    off, col = csr_of_lengths(lengths, Lk, d + 1)
    st = state(len(lengths), d, dtype)
    capi.forward_16("csr", q[:len(lengths)], k, v, *st, row_off=dev(off), col_ind=dev(col)[:300])
    close(st, orc.csr_forward(Qr[:len(lengths)], Kr, Vr, off, col), TOL[dtype], f"short nnz {dtype} d={d}")


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("d", [32, 64, 128])
@pytest.mark.parametrize("L,w,dil,lo,hi", [
    (33, 32, 0, 0, 33), (64, 63, 0, 0, 64), (128, 40, 0, 0, 128), (129, 32, 0, 0, 129), (700, 33, 0, 0, 700),
    (1000, 999, 0, 0, 1000), (1003, 200, 0, 131, 777), (515, 32, 2, 0, 515), (1201, 100, 6, 37, 1200), (300, 299, 15, 0, 300)])
def test_16bit_band_tiles(capi, orc, dtype, d, L, w, dil, lo, hi):
    """Tensor-core band on 16-bit tensors: ragged tiles, one row beyond a tile, row ranges, residue classes; a second call on
    the same state (old rows are merged) and a state with one dead row among fresh ones. The oracle sees the rounded
    tensors; the result's error is the rounding of the stored values."""
    kind, p = ("local_1d_dilated", (w, dil)) if dil else ("local", (w, 0))
    q, k, v = (dev(x).to(dtype) for x in seeded_qkv(L, d, 5 + d))
    Qr, Kr, Vr = (x.float().cpu().numpy() for x in (q, k, v))
    want = orc.implicit_forward(kind, Qr[lo:hi], Kr, Vr, *p, row_begin=lo, row_end=hi)
    st = state(hi - lo, d, dtype)
    st[2].fill_(3.0)  # l = 0: what O holds does not count
    run = lambda s: capi.forward_16(kind, q[lo:hi], k, v, *s, p0=p[0], p1=p[1], row_begin=lo, row_end=hi, tiled=True)
    run(st)
    close(st, want, TOL[dtype], f"{kind} {dtype} L={L} d={d} w={w} dil={dil}")
    # the same keys once more: m and O stay, l doubles; rows whose state was emptied in between give the first result again
    st[0][::5], st[1][::5] = float("-inf"), 0.0
    run(st)
    l2 = 2 * want[1]
    l2[::5] = want[1][::5]
    close(st, (want[0], l2, want[2]), 2 * TOL[dtype], f"{kind} again")


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("d", [32, 128])
@pytest.mark.parametrize("gap", [1, 12, 19, 26])
def test_16bit_band_far_keys_count(capi, orc, dtype, d, gap):
    """A few keys of each window hold almost all of the weight, the 600 others 2^-gap of one of them each. V lets those add up
    to half of the result, or is as large as float16 allows: their probabilities must not fade. Their p is a power of two up
    to the rounding of the scores (2^-11 of gap * ln 2 at most 18, so 1 % at gap 26, where float16 keeps steps of 2^-31)."""
    L, w = 700, 300
    q, k = torch.zeros(L, d), torch.zeros(L, d)
    q[:, 0] = 1.0
    peak = torch.arange(L) % 200 == 77
    k[peak, 0] = gap * float(np.log(2.0)) * d ** 0.5
    far = min(2.0 ** gap / 600, 6.0e4)
    v = torch.where(peak, 1.0, far)[:, None] * torch.linspace(0.5, 1.0, d)
    q, k, v = (x.to(dtype).cuda() for x in (q, k, v))
    want = orc.implicit_forward("local", *(x.float().cpu().numpy() for x in (q, k, v)), w)
    st = state(L, d, dtype)
    capi.forward_16("local", q, k, v, *st, p0=w, tiled=True)
    got = st[2].double().cpu().numpy()
    assert np.max(np.abs(got - want[2]) / np.abs(want[2])) <= TOL[dtype], gap


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("d,w,dil", [(32, 40, 0), (64, 200, 0), (128, 64, 0), (64, 33, 2)])
def test_16bit_band_infinite_values(capi, orc, dtype, d, w, dil):
    """An infinity in V reaches every row whose window holds its key, with its sign; two of opposite signs and NaN give NaN.
    Rows without the key keep their value, except that those of the same tiles may read NaN (0 * inf)."""
    L, s = 600, dil + 1
    kind, p = ("local_1d_dilated", (w, dil)) if dil else ("local", (w,))
    q, k, v = (dev(x).to(dtype) for x in seeded_qkv(L, d, 9 + d))
    for j, c, x in ((300, 0, "inf"), (301, 1, "-inf"), (300, 5, "inf"), (300 + s, 5, "-inf"), (310, d - 1, "nan")):
        v[j, c] = float(x)
    clean = torch.where(torch.isfinite(v), v, torch.zeros_like(v))
    Qr, Kr, Vr, Vc = (x.float().cpu().numpy() for x in (q, k, v, clean))
    want = orc.implicit_forward(kind, Qr, Kr, Vc, *p)
    st = state(L, d, dtype)
    for again in (False, True):  # into an empty state, then merged with what it gave
        capi.forward_16(kind, q, k, v, *st, p0=w, p1=dil, tiled=True)
        got = st[2].double().cpu().numpy()
        i = np.arange(L)
        has = {j: (np.abs(i - j) <= w * s) & ((i - j) % s == 0) for j in (300, 301, 300 + s, 310)}
        both = has[300] & has[300 + s]
        assert np.all(got[has[300], 0] == np.inf) and np.all(got[has[301], 1] == -np.inf)
        assert np.all(np.isnan(got[both, 5])) and np.all(np.isnan(got[has[310], d - 1]))
        assert np.all(got[has[300] & ~both, 5] != -np.inf) and np.all(got[has[300 + s] & ~both, 5] != np.inf)
        for c in range(d):
            reach = {0: has[300], 1: has[301], 5: has[300] | has[300 + s], d - 1: has[310]}.get(c, np.zeros(L, bool))
            rest = got[~reach, c]
            fin = np.isfinite(rest)
            assert np.all(np.isnan(rest[~fin])) and (c in (0, 1, 5, d - 1) or fin.all())
            assert np.max(np.abs(rest - want[2][~reach, c])[fin], initial=0.0) <= (2 if again else 1) * TOL[dtype], c
            near = (np.abs(i - 300) < (w + 2 * 128 + 64) * s) | reach
            assert np.all(np.isfinite(got[~near, c]))


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("d", [32, 64, 128, 40])
@pytest.mark.parametrize("L,w,G,lo,hi", [
    (1500, 20, [0, 1, 2, 3, 4, 5, 6], 0, 1500), (1500, 700, [1499, 3, 3, 800, 0, 800], 0, 1500), (300, 299, [7, 9], 0, 300),
    (2100, 5, [100, 101, 99, 1700, 2099], 100, 1701), (40, 0, list(range(40)), 0, 40)])
def test_16bit_listed_rows(capi, orc, dtype, d, L, w, G, lo, hi):
    """Listed rows have CTAs of their own: side by side, named twice, out of order, outside the row range, without any key
    (window over everything), all rows listed; a second call on the same state."""
    q, k, v = (dev(x).to(dtype) for x in seeded_qkv(L, d, 31 + d))
    Qr, Kr, Vr = (x.float().cpu().numpy() for x in (q, k, v))
    m, l, O = orc.implicit_forward("global_no_local", Qr[lo:hi], Kr, Vr, w, G=np.array(G, dtype=np.int32), row_begin=lo, row_end=hi)
    st = state(hi - lo, d, dtype)
    for times in (1, 2):
        capi.forward_16("global_no_local", q[lo:hi], k, v, *st, global_inds=dev(np.array(G, dtype=np.int32)), p0=w,
                        row_begin=lo, row_end=hi)
        close(st, (m, times * l, O), times * TOL[dtype], f"{dtype} d={d} call {times}")


def test_16bit_listed_rows_side_by_side_run_side_by_side(capi):
    """Sixteen leading listed rows belong to four times as many CTAs as four of them: about the same time, not four times."""
    L, d = 140000, 32
    q, k, v = (torch.randn(L, d, device="cuda").half() for _ in range(3))
    st = state(L, d, torch.float16)

    def ms(n):
        G = torch.arange(n, dtype=torch.int32, device="cuda")
        best = float("inf")
        for _ in range(4):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            capi.forward_16("global_no_local", q, k, v, *st, global_inds=G, p0=16)
            b.record()
            torch.cuda.synchronize()
            best = min(best, a.elapsed_time(b))
        return best

    four, sixteen = ms(4), ms(16)
    assert sixteen < 2 * four, (four, sixteen)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("dil", [0, 2])
def test_16bit_window_routes_of_the_modules(pkg, capi, orc, dtype, dil):
    """The modules hand wide 16-bit windows to the tensor-core kernel as they are (no tensor is allocated) and convert where
    TMA cannot address a tensor or where the state overlaps an input; both give the same window."""
    L, d, w = 500, 64, 40
    mod = pkg.binding("spfa_local_1d_dilated" if dil else "spfa_local")
    args = (w, dil) if dil else (w,)
    q, k, v = (dev(x).to(dtype) for x in seeded_qkv(L, d, 3))
    want = orc.implicit_forward("local_1d_dilated" if dil else "local", *(x.float().cpu().numpy() for x in (q, k, v)), *args)

    def run(q, k, v, st):
        n = torch.cuda.memory_stats()["allocation.all.allocated"]
        mod.forward(q, k, v, *st, *args)
        n = torch.cuda.memory_stats()["allocation.all.allocated"] - n
        close(st, want, TOL[dtype], f"{dtype} dil={dil}")
        return n

    run(q, k, v, state(L, d, dtype))
    assert run(q, k, v, state(L, d, dtype)) == 0
    odd = torch.empty(L * d + 1, dtype=dtype, device="cuda")[1:].view(L, d).copy_(k)  # 2 bytes off a 16-byte boundary
    assert run(q, odd, v, state(L, d, dtype)) > 0
    m, l, _ = state(L, d, dtype)
    own = q.clone()
    assert run(own, k, v, (m, l, own)) > 0  # O is Q: read before it is written


def test_16bit_window_rule(capi):
    usable = capi.lib().spfa_tiled_16_usable
    assert [usable(t, 64, w, 1) for t in (1, 2) for w in (31, 32, (1 << 17) - 1, 1 << 17)] == [0, 1, 1, 0, 0, 1, 1, 1]
    assert [usable(1, d, 64, s) for d, s in ((48, 1), (64, 16), (64, 17), (64, 0))] == [0, 1, 0, 0]
    capi.set_path(capi.PATH_GATHER)
    assert usable(1, 64, 64, 1) == 0


@pytest.mark.parametrize("d", [32, 64, 128])
@pytest.mark.parametrize("fault", ["none", "unsorted", "beyond"])
def test_scattered_blocks_of_an_explicit_mask(capi, orc, d, fault):
    """Row blocks without a dense tile are copied whole: empty rows at block ends, rows around the listing (128) and slicing
    (1024) limits, a row whose last column exceeds the next row's first; with a row out of order or a column beyond the keys
    (dropped) in the second block; then the same plan over two key ranges."""
    Lk = 200000
    lengths = [0] + [5] * 60 + [127, 128, 129, 1023, 1024, 1025, 2500] + [40] * 59 + [0] + [33] * 70 + [0] * 3 + [1] * 72
    off, col = csr_of_lengths(lengths, Lk, d)
    n, at = len(lengths), int(off[150])
    rows = np.repeat(np.arange(n), lengths)
    sampled = rows % 4 == 0  # a tile is dense from 128 * 64 / 24 entries on, a quarter of them in every fourth row
    assert n > 256 and np.unique(rows[sampled] // 128 * Lk + col[sampled] // 64, return_counts=True)[1].max() < 128 * 64 / 24 / 4
    if fault == "unsorted":
        col[at], col[at + 1] = col[at + 1], col[at]
    if fault == "beyond":
        col[at] = Lk + 7
    Q, K, V = seeded_qkv(n, d, 3 + d, Lk=Lk)
    want = orc.csr_forward(Q, K, V, off, col, use_nan=True)
    q, k, v = dev(Q), dev(K), dev(V)
    capi.set_path(capi.PATH_TILED)
    st = state(n, d, torch.float32)
    capi.csr_forward(q, k, v, dev(off), dev(col), *st, use_nan=True)
    assert capi.last_path() == capi.PATH_TILED
    close(st, want, TOL[torch.float32], f"one call, d={d}, {fault}")
    plan = capi.csr_plan(dev(off), dev(col), Lk, d)
    st = state(n, d, torch.float32)
    capi.planned_forward_keys(q, k, v, *st, plan, 0, 64 * 1500, use_nan=True)
    capi.planned_forward_keys(q, k, v, *st, plan, 64 * 1500, Lk)
    close(st, want, TOL[torch.float32], f"two ranges, d={d}, {fault}")
