"""attention (head 128), the step after the 'heads' projection: the reference's cases (test/kernels.test.js:148-165) and wider ones,
through the C ABI against the CPU restatement of cpuAttn."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ATT = [   # test/kernels.test.js:149-151
    dict(label="no mask", Hq=2, Hkv=2, Lq=96, Lk=96, mode=0),
    dict(label="causal + valid length 80, GQA 4:2", Hq=4, Hkv=2, Lq=96, Lk=96, mode=1, nvalid=80),
    dict(label="valid length 77 of 100 keys, 64 queries", Hq=2, Hkv=2, Lq=64, Lk=100, mode=2, nvalid=77),
]
MORE = [
    dict(label="ragged tiles, GQA 6:2", Hq=6, Hkv=2, Lq=150, Lk=333, mode=0),
    dict(label="causal, long", Hq=2, Hkv=1, Lq=300, Lk=300, mode=1, nvalid=300),
    dict(label="one query", Hq=3, Hkv=3, Lq=1, Lk=70, mode=2, nvalid=33),
    dict(label="custom scale, output row stride", Hq=2, Hkv=2, Lq=70, Lk=130, mode=0, scale=0.05, ldo=2 * 128 + 64),
]


WIDE = [   # several blocks of two 128-query tiles, key tiles of 128, a last block with one tile, ragged ends
    dict(label="700 x 700, causal + valid length 650", Hq=2, Hkv=1, Lq=700, Lk=700, mode=1, nvalid=650),
    dict(label="384 x 520, GQA 4:2", Hq=4, Hkv=2, Lq=384, Lk=520, mode=0),
    dict(label="257 x 1000, valid length 901", Hq=2, Hkv=2, Lq=257, Lk=1000, mode=2, nvalid=901),
    dict(label="wide score range (the running maximum moves by more than the lazy threshold)", Hq=2, Hkv=2, Lq=300, Lk=640, mode=0, qstd=4.0),
    dict(label="512 x 512, output rows not 16-byte aligned", Hq=1, Hkv=1, Lq=512, Lk=512, mode=0, ldo=128 + 6),
]


@pytest.mark.parametrize("kernel", ["warp", "tmem"])
@pytest.mark.parametrize("c", ATT + MORE + WIDE, ids=lambda c: c["label"])
def test_attention_head128(gpu, oracle, c, kernel):
    import p0pc0rn_kernels_b200 as P
    O = oracle
    D, Hq, Hkv, Lq, Lk = 128, c["Hq"], c["Hkv"], c["Lq"], c["Lk"]
    Q = O.round_f16(O.randn(Hq * Lq * D, 21, c.get("qstd", 0.5))); Kt = O.round_f16(O.randn(Hkv * Lk * D, 22, 0.5)); V = O.round_f16(O.randn(Hkv * Lk * D, 23))
    ldo = c.get("ldo", Hq * D)
    qb, kb, vb = gpu.upload(P.toF16(Q)), gpu.upload(P.toF16(Kt)), gpu.upload(P.toF16(V))
    ob = gpu.upload(np.full(Lq * ldo, 0x7E01, np.uint16))                                    # NaN poison: only the head columns may change
    try:
        a = {"q": {"buf": qb}, "k": {"buf": kb}, "v": {"buf": vb}, "o": {"buf": ob, "ld": ldo}, "Lq": Lq, "Lk": Lk, "Hq": Hq, "Hkv": Hkv,
             "mode": c["mode"], "nvalid": c.get("nvalid"), "kernel": kernel}
        if "scale" in c: a["scale"] = c["scale"]
        fl = P.attention(gpu, a)
        assert fl == 4.0 * Lq * Lk * 128 * Hq
        assert gpu.lastKernel == {"warp": 16, "tmem": 17}[kernel]
        raw = gpu.read(ob, 0, Lq * ldo * 2).view(np.uint16).reshape(Lq, ldo)
        assert (raw[:, Hq * D:] == 0x7E01).all(), "columns past the heads were written"
        got = P.fromF16(np.ascontiguousarray(raw[:, :Hq * D]).ravel())
        want = O.cpu_attn(Q, Kt, V, Hq=Hq, Hkv=Hkv, Lq=Lq, Lk=Lk, mode=c["mode"], nvalid=c.get("nvalid"), scale=c.get("scale"))
        cos, maxabs = O.compare(got, want)[:2]
        assert cos > 0.9995, (cos, maxabs)                                                      # the reference's gate (test/kernels.test.js:228)
        assert np.abs(got - want).max() <= 2e-2 * np.abs(want).max()
    finally:
        for b in (qb, kb, vb, ob): gpu.free(b)


def test_attention_dit_shape(gpu, oracle):
    """24 heads x 3600 tokens (the attention after the DiT projection): the library's own choice of kernel, two heads checked."""
    import p0pc0rn_kernels_b200 as P
    O = oracle
    D, H, L = 128, 24, 3600
    Q = O.round_f16(O.randn(H * L * D, 31, 0.5)); Kt = O.round_f16(O.randn(H * L * D, 32, 0.5)); V = O.round_f16(O.randn(H * L * D, 33))
    qb, kb, vb, ob = gpu.upload(P.toF16(Q)), gpu.upload(P.toF16(Kt)), gpu.upload(P.toF16(V)), gpu.buffer(L * H * D * 2)
    try:
        P.attention(gpu, {"q": {"buf": qb}, "k": {"buf": kb}, "v": {"buf": vb}, "o": {"buf": ob}, "Lq": L, "Lk": L, "Hq": H, "Hkv": H, "mode": 0})
        assert gpu.lastKernel == 17
        got = P.fromF16(gpu.read(ob, 0, L * H * D * 2).view(np.uint16)).reshape(L, H, D)
        assert np.isfinite(got).all()
        for h in (0, 23):
            sl = slice(h * L * D, (h + 1) * L * D)
            want = O.cpu_attn(Q[sl], Kt[sl], V[sl], Hq=1, Hkv=1, Lq=L, Lk=L, mode=0).reshape(L, D)
            cos = O.compare(got[:, h].ravel(), want.ravel())[0]
            assert cos > 0.9995, (h, cos)
            assert np.abs(got[:, h] - want).max() <= 2e-2 * np.abs(want).max()
    finally:
        for b in (qb, kb, vb, ob): gpu.free(b)


def test_attention_errors(gpu):
    import p0pc0rn_kernels_b200 as P
    b = gpu.buffer(1024)
    with pytest.raises(ValueError, match="needs"):
        P.attention(gpu, {"q": {"buf": b}, "k": {"buf": b}, "v": {"buf": b}, "o": {"buf": b}, "Lq": 64, "Lk": 64, "Hq": 2})
    with pytest.raises(ValueError, match="multiple of Hkv"):
        P.attention(gpu, {"q": {"buf": b}, "k": {"buf": b}, "v": {"buf": b}, "o": {"buf": b}, "Lq": 1, "Lk": 1, "Hq": 3, "Hkv": 2})
    gpu.free(b)


@pytest.mark.parametrize("Hq,Hkv,Lq,Lk,mode,nvalid", [
    (4, 1, 4, 64, 0, 64),         # 16 packed rows: one full row tile, one key tile, no split
    (17, 1, 1, 65, 0, 65),        # 17 rows: two row tiles, a last key tile of one key
    (8, 2, 8, 700, 2, 641),       # 32 rows, splits whose last tile holds one valid key
    (3, 1, 11, 1000, 2, 640),     # 33 rows: four row tiles, the last one with one row; splits that end on a tile's edge
    (8, 1, 9, 2000, 2, 1999),     # 72 rows: two row blocks
    (2, 2, 100, 300, 1, 90),      # causal: rows that see fewer keys than the first split holds, row blocks with their own key counts
    (32, 8, 1, 4096, 2, 4000),    # a decoding step: 16 splits and more, merged by the last block
])
def test_attention_split_keys(gpu, oracle, Hq, Hkv, Lq, Lk, mode, nvalid):
    """the split-key kernel of short query runs, at the edges of its row tiles, key tiles and splits; twice, so that a counter left
    over from the first call would show"""
    import p0pc0rn_kernels_b200 as P
    O = oracle
    Q = O.round_f16(O.randn(Hq * Lq * 128, 21, 0.5)); Kt = O.round_f16(O.randn(Hkv * Lk * 128, 22, 0.5)); V = O.round_f16(O.randn(Hkv * Lk * 128, 23))
    want = O.cpu_attn(Q, Kt, V, Hq=Hq, Hkv=Hkv, Lq=Lq, Lk=Lk, mode=mode, nvalid=nvalid)
    kh = P.toF16(Kt).reshape(Hkv, Lk, 128); vh = P.toF16(V).reshape(Hkv, Lk, 128)
    if mode == 2: kh[:, nvalid:] = 0x7E01; vh[:, nvalid:] = 0x7E01                            # the unused end of a cache may hold anything, NaN too
    qb, kb, vb = gpu.upload(P.toF16(Q)), gpu.upload(kh), gpu.upload(vh)
    ob = gpu.buffer(Lq * Hq * 256)
    try:
        for _ in range(2):
            gpu.upload(np.full(Lq * Hq * 128, 0x7E01, np.uint16), dst=ob)
            P.attention(gpu, {"q": {"buf": qb}, "k": {"buf": kb}, "v": {"buf": vb}, "o": {"buf": ob}, "Lq": Lq, "Lk": Lk, "Hq": Hq, "Hkv": Hkv, "mode": mode, "nvalid": nvalid})
            assert gpu.lastKernel == 16
            got = P.fromF16(gpu.read(ob).view(np.uint16))
            assert O.compare(got, want)[0] > 0.9995
            assert np.abs(got - want).max() <= 2e-2 * np.abs(want).max()
    finally:
        for b in (qb, kb, vb, ob): gpu.free(b)


@pytest.mark.parametrize("Lk,splits", [(60, False), (4096, True)])
def test_attention_split_keys_special_values(gpu, Lk, splits):
    """keys of score minus infinity weigh nothing (two whole key tiles of them: a share, or a split, that saw no other), a NaN among the valid keys
    reaches every row that sees it and no other, an infinite value its own column"""
    import p0pc0rn_kernels_b200 as P
    rng = np.random.default_rng(5)
    Hq, Hkv, nv = 12, 3, Lk - 3
    q = rng.normal(0, 0.5, (Hq, 1, 128)); k = rng.normal(0, 0.5, (Hkv, Lk, 128)); v = rng.normal(0, 1, (Hkv, Lk, 128))
    q[:, :, 0] = 0.5
    gone = slice(128, 256) if splits else slice(16, 48)
    k[0, gone, 0] = -np.inf
    k[1, nv - 2, 3] = np.nan
    v[2, 7, 5] = np.inf
    q, k, v = (t.astype(np.float16) for t in (q, k, v))
    k[:, nv:] = np.nan; v[:, nv:] = np.nan                                                    # past the valid length: never read
    with np.errstate(invalid="ignore"):
        s = np.einsum("hqd,hkd->hqk", q.astype(np.float64), np.repeat(k, Hq // Hkv, 0).astype(np.float64)[:, :nv]) / 128 ** 0.5
        p = np.exp(s - s.max(2, keepdims=True)); p /= p.sum(2, keepdims=True)
        want = np.einsum("hqk,hkd->qhd", p, np.repeat(v, Hq // Hkv, 0).astype(np.float64)[:, :nv])[0]
    qb, kb, vb, ob = gpu.upload(q), gpu.upload(k), gpu.upload(v), gpu.buffer(Hq * 256)
    try:
        P.attention(gpu, {"q": {"buf": qb}, "k": {"buf": kb}, "v": {"buf": vb}, "o": {"buf": ob}, "Lq": 1, "Lk": Lk, "Hq": Hq, "Hkv": Hkv, "mode": 2, "nvalid": nv})
        assert gpu.lastKernel == 16 and (gpu.lastPlan["S"] > 1) == splits
        got = P.fromF16(gpu.read(ob).view(np.uint16)).reshape(Hq, 128)
        assert np.isnan(got[4:8]).all() and np.isfinite(got[:4]).all()
        assert np.array_equal(np.isposinf(got[8:]), np.isposinf(want[8:])) and np.isposinf(got[8:, 5]).all() and not np.isnan(got[8:]).any()
        f = np.isfinite(want) & np.isfinite(got)
        assert np.abs(got[f] - want[f]).max() <= 2e-2 * np.abs(want[f]).max()
    finally:
        for b in (qb, kb, vb, ob): gpu.free(b)


def test_attention_split_keys_many_row_blocks(gpu):
    """more blocks of 64 query rows than a grid has in y or z (forced: the library's own choice for so many queries is the other kernel)"""
    import torch

    import p0pc0rn_kernels_b200 as P
    Lq, Lk = 64 * 65536 + 5, 65
    g = torch.Generator(device="cuda"); g.manual_seed(1)
    q, k, v = (torch.empty(n, 128, device="cuda", dtype=torch.float16).normal_(0, 0.5, generator=g) for n in (Lq, Lk, Lk))
    o = torch.full((Lq, 128), float("nan"), device="cuda", dtype=torch.float16)
    torch.cuda.synchronize()
    bufs = [gpu.wrap(t.data_ptr(), t.numel() * 2) for t in (q, k, v, o)]
    try:
        P.attention(gpu, {**{n: {"buf": b} for n, b in zip("qkvo", bufs)}, "Lq": Lq, "Lk": Lk, "Hq": 1, "mode": 0, "kernel": "warp"})
        gpu.done()
        assert gpu.lastPlan["row_blocks"] == 65537
        for r0 in (0, 64 * 32767, 64 * 65535, Lq - 69):
            want = torch.softmax(q[r0:r0 + 69].float() @ k.float().T / 128 ** 0.5, -1) @ v.float()
            assert (o[r0:r0 + 69].float() - want).abs().max() <= 2e-2 * want.abs().max()
        assert torch.isfinite(o).all()
    finally:
        for b in bufs: gpu.free(b)
        del q, k, v, o
        torch.cuda.empty_cache()


def test_split_calls_recorded_first(gpu, oracle):
    """recorded before the context has any scratch memory: attention that would split its keys runs unsplit (and says so), a multiply that
    splits k is refused, and after one eager call both record as they run eagerly"""
    import p0pc0rn_kernels_b200 as P
    O = oracle
    Hq, Hkv, Lk, N, K, M = 8, 2, 1000, 256, 4096, 64
    Q = O.round_f16(O.randn(Hq * 128, 21, 0.5)); Kt = O.round_f16(O.randn(Hkv * Lk * 128, 22, 0.5)); V = O.round_f16(O.randn(Hkv * Lk * 128, 23))
    X = O.round_f16(O.randn(M * K, 24)); W = O.round_f16(O.randn(N * K, 25, 0.02))
    own = P.createGpu({"device": 0})
    qb, kb, vb, xb, wb = own.upload(P.toF16(Q)), own.upload(P.toF16(Kt)), own.upload(P.toF16(V)), own.upload(P.toF16(X)), own.upload(P.toF16(W))
    ob, yb = own.buffer(Hq * 256), own.buffer(M * N * 4)
    plans = []

    def attn():
        P.attention(own, {"q": {"buf": qb}, "k": {"buf": kb}, "v": {"buf": vb}, "o": {"buf": ob}, "Lq": 1, "Lk": Lk, "Hq": Hq, "Hkv": Hkv, "mode": 0})
        plans.append(own.lastPlan["S"])

    def mul():
        P.gemm(own, {"w": {"enc": "f16", "buf": wb, "off": 0, "rows": N, "cols": K}, "x": {"buf": xb}, "y": {"buf": yb}, "M": M, "N": N, "K": K, "epi": "f32"})
        plans.append(own.lastPlan["S"])

    def check():
        got = P.fromF16(own.read(ob).view(np.uint16)); want = O.cpu_attn(Q, Kt, V, Hq=Hq, Hkv=Hkv, Lq=1, Lk=Lk, mode=0, nvalid=Lk)
        assert np.abs(got - want).max() <= 2e-2 * np.abs(want).max()
    graphs = []
    try:
        graphs.append(own.record(attn)); graphs[0].launch()
        check()
        assert plans == [1]
        with pytest.raises(ValueError, match="run it once before"):
            own.record(mul)
        assert not own.lost
        attn(); mul()
        eager = own.read(ob).tobytes() + own.read(yb).tobytes()
        graphs.append(own.record(lambda: (attn(), mul())))
        assert plans[1:3] == plans[3:] and min(plans[1:3]) > 1, plans
        own.upload(np.zeros(Hq * 128, np.uint16), "", ob, 0); own.upload(np.zeros(M * N, np.float32), "", yb, 0)
        graphs[1].launch()
        assert own.read(ob).tobytes() + own.read(yb).tobytes() == eager
        check()
        y = own.read(yb).view(np.float32).reshape(M, N); ref = X.reshape(M, K).astype(np.float64) @ W.reshape(N, K).astype(np.float64).T
        assert np.linalg.norm(y - ref) <= 1e-5 * np.linalg.norm(ref)
    finally:
        for g in graphs: g.free()
        for b in (qb, kb, vb, xb, wb, ob, yb): own.free(b)
        own.close()
