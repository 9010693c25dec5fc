"""Numerics of every CUDA kernel against a plain PyTorch fp32 reference of the same op."""
import math

import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def C():
    from flodl_b200 import _ext
    return _ext.require()


def _ref_gemm(a, b, a_mn, b_mn):
    A = a.float().t() if a_mn else a.float()
    B = b.float().t() if b_mn else b.float()
    return A @ B.t()


def _gemm_case(C, M, N, K, a_mn, b_mn, config, out_dtype=torch.bfloat16, **kw):
    torch.manual_seed(M * 7 + N * 3 + K)
    dev = "cuda"
    a = torch.randn((K, M) if a_mn else (M, K), device=dev).bfloat16()
    b = torch.randn((K, N) if b_mn else (N, K), device=dev).bfloat16()
    out = torch.zeros(M, N, device=dev, dtype=out_dtype)
    C.clear_status(0)
    C.gemm(a, b, out, a_mn, b_mn, config=config, **kw)
    torch.cuda.synchronize()
    assert C.read_status(0) == 0, f"kernel status {C.read_status(0)}"
    ref = _ref_gemm(a, b, a_mn, b_mn)
    return out.float(), ref


@pytest.mark.parametrize("config", [2, 1, 3, 0, 4])
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True)])
def test_gemm_layouts(C, config, a_mn, b_mn):
    out, ref = _gemm_case(C, 512, 768, 256, a_mn, b_mn, config)
    err = (out - ref).abs().max().item()
    assert err <= 0.02 * ref.abs().max().item() + 0.05, f"max err {err}"


@pytest.mark.parametrize("config", [0, 1, 2, 3, 4, 5])
def test_gemm_ragged_edges(C, config):
    # M, N not multiples of the tile, K not a multiple of 64 (TMA zero-fills the tails)
    out, ref = _gemm_case(C, 300, 328, 200, False, False, config)
    err = (out - ref).abs().max().item()
    assert err <= 0.02 * ref.abs().max().item() + 0.05, f"max err {err}"


@pytest.mark.parametrize("config", [0, 2, 4, 5])
def test_gemm_many_tiles_per_cta(C, config):
    # more tiles than SMs: exercises the accumulator double buffering and barrier phases
    out, ref = _gemm_case(C, 4096, 3072, 768, False, False, config)
    err = (out - ref).abs().max().item()
    assert err <= 0.02 * ref.abs().max().item() + 0.05, f"max err {err}"


@pytest.mark.parametrize("config", [-1, 0, 1, 4, 5])
def test_gemm_bias_gelu_aux(C, config):
    M, N, K = 512, 768, 256
    torch.manual_seed(0)
    a = torch.randn(M, K, device="cuda").bfloat16()
    b = (torch.randn(N, K, device="cuda") / math.sqrt(K)).bfloat16()
    bias = torch.randn(N, device="cuda")
    out = torch.empty(M, N, device="cuda", dtype=torch.bfloat16)
    aux = torch.empty_like(out)
    C.gemm(a, b, out, bias=bias, epi=1, aux=aux, config=config)
    pre = a.float() @ b.float().t() + bias
    ref = torch.nn.functional.gelu(pre)
    assert (aux.float() - pre).abs().max().item() < 0.05
    assert (out.float() - ref).abs().max().item() < 0.05
    # backward epilogue: dY * gelu'(aux)
    g = torch.randn(M, K, device="cuda").bfloat16()
    w = (torch.randn(N, K, device="cuda") / math.sqrt(K)).bfloat16()
    dpre = torch.empty(M, N, device="cuda", dtype=torch.bfloat16)
    C.gemm(g, w, dpre, epi=2, aux=aux, config=config)
    x = aux.float().requires_grad_(True)
    torch.nn.functional.gelu(x).backward(g.float() @ w.float().t())
    assert (dpre.float() - x.grad).abs().max().item() < 0.06


@pytest.mark.parametrize("config", [0, 1, 2, 3, 4, 5])
@pytest.mark.parametrize("M,N,K,pad,bias", [(300, 328, 64, 0, "fp32"), (513, 1160, 72, 8, "bf16"), (2500, 2824, 128, 0, "offset"), (129, 72, 200, 4, "none")])
def test_gemm_staged_epilogues(C, config, M, N, K, pad, bias):
    """Scale, bias, GELU with its pre-activation and GELU' where tiles are ragged, a CTA has several of them, rows of `aux` are not 16-byte aligned, the bias
    is of either type and starts anywhere. Bounds: one rounding to bf16 (2^-8 of the value) plus 3e-4 of the factor's scale for the hardware's tanh."""
    torch.manual_seed(M + config)
    a = torch.randn(M, K, device="cuda").bfloat16()
    b = (torch.randn(N, K, device="cuda") / math.sqrt(K)).bfloat16()
    v = {"fp32": torch.randn(N, device="cuda"), "bf16": torch.randn(N, device="cuda").bfloat16(), "offset": torch.randn(N + 1, device="cuda")[1:], "none": None}[bias]
    lin = a.double() @ b.double().t()
    pre = lin + (0 if v is None else v.double())

    def close(got, want, scale=1.0, tail=3e-4):
        assert C.read_status(0) == 0
        assert ((got.double() - want).abs() <= want.abs() * 2.0 ** -8 + tail * scale + 1e-4).all()
    C.clear_status(0)
    out = torch.empty(M, N, device="cuda", dtype=torch.bfloat16)
    C.gemm(a, b, out, bias=v, config=config)
    close(out, pre)
    alpha = torch.tensor([-0.5], device="cuda")
    out32 = torch.ones(M, N, device="cuda")
    C.gemm(a, b, out32, bias=v, config=config, alpha=alpha, accumulate=True)
    close(out32, 1 - 0.5 * lin + (0 if v is None else v.double()))
    for tanh in (False, True):
        aux = torch.full((M, N + pad), 9.0, device="cuda", dtype=torch.bfloat16)
        C.gemm(a, b, out, bias=v, epi=3 if tanh else 1, aux=aux[:, :N], config=config)
        close(aux[:, :N], pre)
        assert (aux[:, N:] == 9).all()
        close(out, F.gelu(pre, approximate="tanh" if tanh else "none"), pre.abs() + 1)
        C.gemm(a, b, out, bias=v, epi=3 if tanh else 1, config=config)
        close(out, F.gelu(pre, approximate="tanh" if tanh else "none"), pre.abs() + 1)
        aux[0, 0], aux[M - 1, N - 1], aux[M - 1, 0] = float("nan"), 40.0, -40.0
        x = aux[:, :N].double().requires_grad_()
        F.gelu(x, approximate="tanh" if tanh else "none").sum().backward()
        dpre = torch.empty_like(out)
        C.gemm(a, b, dpre, epi=4 if tanh else 2, aux=aux[:, :N], config=config)
        assert dpre[0, 0].isnan()
        dpre[0, 0] = x.grad[0, 0] = 0
        close(dpre, lin * x.grad, lin.abs() + 1)


@pytest.mark.parametrize("rows,n,k,epi,bias", [(4096, 768, 768, 0, True), (3054, 768, 3072, 2, True), (2500, 2304, 768, 0, False), (8192, 520, 1032, 4, True),
                                               (20000, 264, 256, 0, True), (1030, 2056, 264, 0, True), (3400, 2312, 264, 0, True), (256, 8, 8, 0, True),
                                               (65, 72, 40, 2, True), (77, 768, 768, 0, True), (130, 3072, 104, 4, False), (2000, 136, 520, 2, True)])
def test_linear_gradients_in_one_launch(C, rows, n, k, epi, bias):
    """dX, dW and db from one launch where tiles are ragged and the pairs' shares of dW start anywhere in a tile. dX is rounded to bf16 once (and the
    activation's derivative takes the hardware's tanh: 3e-4); dW and db are fp32 sums of exact products."""
    torch.manual_seed(rows + n)
    dy, w, x = (torch.randn(s, device="cuda").bfloat16() for s in ((rows, n), (n, k), (rows, k)))
    dy, w = dy * 0.1, w / math.sqrt(n)
    aux = torch.randn(rows, k, device="cuda").bfloat16() if epi else None
    dx = torch.empty(rows, k, device="cuda", dtype=torch.bfloat16)
    dw, db = torch.randn(n, k, device="cuda"), torch.randn(n, device="cuda")
    want_dw, want_db = dw.double() + dy.double().t() @ x.double(), db.double() + dy.double().sum(0)
    lin = want = dy.double() @ w.double()
    if epi:
        h = aux.double().requires_grad_()
        F.gelu(h, approximate="none" if epi == 2 else "tanh").sum().backward()
        want = lin * h.grad
    C.clear_status(0)
    assert C.gemm_backward(dy, w, x, dx, dw, db if bias else None, epi, aux)
    assert C.read_status(0) == 0
    assert ((dx.double() - want).abs() <= want.abs() * 2.0 ** -8 + (3e-4 if epi else 0) * (lin.abs() + 1) + 1e-5).all()
    # fp32 sums over `rows` terms: a few ulp of the sum of magnitudes
    assert ((dw.double() - want_dw).abs() <= 2.0 ** -20 * (dy.double().abs().t() @ x.double().abs() + 8)).all()
    if bias:
        assert ((db.double() - want_db).abs() <= 2.0 ** -20 * (dy.double().abs().sum(0) + 8)).all()


def test_copy_buffers(C):
    """Bytes arrive as they are at every length and alignment; what is not a plain copy on one device is refused, with nothing done."""
    src = [torch.randint(0, 256, (n,), device="cuda", dtype=torch.uint8) for n in (1, 15, 16, 16383, 16384, 16385, 100003)] + [torch.randn(3, 0, device="cuda")]
    dst = [torch.zeros_like(s) for s in src]
    assert C.copy_buffers(dst, src) and all(torch.equal(d, s) for d, s in zip(dst, src))
    odd = [torch.zeros(40001, device="cuda", dtype=torch.uint8)[1:], torch.zeros(5003, device="cuda", dtype=torch.float32)[3:]]
    new = [torch.randint(0, 256, (40000,), device="cuda", dtype=torch.uint8), torch.randn(5000, device="cuda")]
    assert C.copy_buffers(odd, new) and all(torch.equal(d, s) for d, s in zip(odd, new))
    a, b = torch.zeros(8, 8, device="cuda"), torch.ones(8, 8, device="cuda")
    for d, s in ((a, b.cpu()), (a, b.t()), (a, b[:1]), (a, b.double()), (a, a), (a.view(-1)[:60], a.view(-1)[4:]), (a, b.clone().requires_grad_())):
        assert not C.copy_buffers([d], [s])
    assert not C.copy_buffers([a, a], [b, b]) and not C.copy_buffers([a] * 9, [b] * 9) and not a.any()


@pytest.mark.parametrize("src_at", [0, 1, 2, 4, 6, 8, 12, 16])
@pytest.mark.parametrize("dst_at", [0, 1, 2, 4, 8])
def test_copy_buffers_at_every_alignment(C, src_at, dst_at):
    """Each width of vector, alone and with a rest, around the sizes of a block; bytes before and behind stay."""
    for n in (1, 3, 255, 4099, 16383, 16384, 16385, 65551):
        src, dst = torch.randint(0, 256, (n + 64,), device="cuda", dtype=torch.uint8), torch.full((n + 64,), 7, device="cuda", dtype=torch.uint8)
        assert C.copy_buffers([dst[dst_at:dst_at + n]], [src[src_at:src_at + n]])
        assert torch.equal(dst[dst_at:dst_at + n], src[src_at:src_at + n]) and (dst[:dst_at] == 7).all() and (dst[dst_at + n:] == 7).all()


def test_a_copy_off_alignment_takes_no_longer_than_the_librarys(C):
    """64 MB from an address off a 16-byte boundary, as a slice of a larger tensor has it: as fast as `copy_` within the noise of a shared GPU (byte by byte it was 5 times as long)."""
    n = 64 << 20
    src, dst = torch.zeros(n + 16, device="cuda", dtype=torch.uint8), torch.zeros(n, device="cuda", dtype=torch.uint8)

    def us(call):
        best = float("inf")
        for _ in range(10):
            a, b = torch.cuda.Event(True), torch.cuda.Event(True)
            a.record()
            call()
            b.record()
            b.synchronize()
            best = min(best, a.elapsed_time(b) * 1e3)
        return best
    for at in (8, 4, 2, 1):
        assert us(lambda: C.copy_buffers([dst], [src[at:at + n]])) < 1.5 * us(lambda: dst.copy_(src[at:at + n])), at


def test_dropout_keeps_what_its_threshold_says(C):
    """One draw per value: what a larger p keeps, a smaller one keeps too, in shares of 1 - p (within six standard deviations), also at the ends."""
    x, n = torch.ones(1 << 22, device="cuda"), 1 << 22
    kept = {p: C.dropout(x, p, 11, None) != 0 for p in (0.0, 1e-8, 2.0 ** -24, 0.1, 0.5, 0.9, 1 - 2.0 ** -24)}
    ps = sorted(kept)
    for a, b in zip(ps, ps[1:]):
        assert not (kept[b] & ~kept[a]).any()
    for p in ps:
        assert abs(kept[p].sum().item() - n * (1 - p)) <= 6 * math.sqrt(n * p * (1 - p)) + 1


@pytest.mark.parametrize("rows,V,K,sparse", [(1024, 4104, 200, True), (4096, 8200, 768, True), (1500, 3000, 264, False), (4096, 8200, 264, False)])
def test_linear_cross_entropy_gradients_with_few_rows(monkeypatch, rows, V, K, sparse):
    """The projection's dX, whose reduction over the vocabulary is split where rows make few tiles, and its dW and db. dX is rounded to bf16 once from
    gradients of the logits that are rounded to bf16 (2^-8 each; their errors add like independent ones over V terms)."""
    from flodl_b200 import ops
    from flodl_b200.ops import core
    monkeypatch.setitem(core._EAGER, "min_numel", 0)      # the native kernels at every size, as in a captured step
    torch.manual_seed(V)
    x = torch.randn(rows, K, device="cuda").bfloat16().requires_grad_()
    w = (torch.randn(V, K, device="cuda") * 0.05).bfloat16().requires_grad_()
    b = torch.randn(V, device="cuda").requires_grad_()
    t = torch.randint(0, V, (rows,), device="cuda")
    if sparse:
        t[torch.rand(rows, device="cuda") < 0.85] = -100
    w._fb_grad, b._fb_grad = torch.zeros(V, K, device="cuda"), torch.zeros(V, device="cuda")
    (3.0 * ops.linear_cross_entropy(x, w, b, t, -100, sparse)).backward()
    xd, wd, bd = (v.detach().double().requires_grad_() for v in (x, w, b))
    (3.0 * F.cross_entropy(xd @ wd.t() + bd, t, ignore_index=-100)).backward()
    for got, want in ((x.grad, xd.grad), (w._fb_grad, wd.grad), (b._fb_grad, bd.grad)):
        assert (got.double() - want).norm() <= 0.01 * want.norm()
    assert sparse is False or (x.grad[t == -100] == 0).all()


@pytest.mark.parametrize("config", [0, 1, 2, 3, 4, 5])
@pytest.mark.parametrize("blocks,parts", [(33, 16), (500, 31), (5, 4), (3, 7), (1, 2)])
def test_gemm_split_into_more_parts_than_hold_a_block(C, config, blocks, parts):
    """Equal parts of a reduction, rounded up to whole K blocks, may be over before the last part starts, on the host's sizes or on the device's. fp32 sums of
    exact products: a few ulp of the sum of magnitudes. What an earlier product left in the accumulators must not come in."""
    torch.manual_seed(blocks)
    M, N, K = 300, 328, blocks * 64
    big = torch.full((4096, 64), 1e4, device="cuda").bfloat16()
    a, b, bias = torch.randn(M, K, device="cuda").bfloat16(), torch.randn(N, K, device="cuda").bfloat16(), torch.randn(N, device="cuda")
    C.clear_status(0)
    for k_dyn in (None, 64 * max(1, blocks // 9)):
        k = K if k_dyn is None else k_dyn
        ad, bd = a[:, :k].double(), b[:, :k].double()
        C.gemm(big, big, torch.empty(4096, 4096, device="cuda", dtype=torch.bfloat16), config=config)
        out = torch.ones(M, N, device="cuda")
        C.gemm(a, b, out, bias=bias, accumulate=True, split_k=parts, config=config, k_dyn=None if k_dyn is None else torch.tensor([k], device="cuda", dtype=torch.int32))
        assert C.read_status(0) == 0
        assert ((out.double() - 1 - bias.double() - ad @ bd.t()).abs() <= 2.0 ** -20 * (ad.abs() @ bd.abs().t() + 8)).all()


@pytest.mark.parametrize("rows,V,K,sparse", [(256, 32000, 512, False), (64, 32000, 128, False), (256, 18440, 256, False), (200, 50257, 512, False), (128, 28996, 256, False),
                                             (1024, 32000, 512, True), (1024, 25000, 768, True), (1024, 50257, 512, True)])
def test_linear_cross_entropy_gradients_over_large_vocabularies(C, monkeypatch, rows, V, K, sparse):
    """As above at vocabularies whose K blocks the parts do not divide."""
    big = torch.full((4096, 64), 1e4, device="cuda").bfloat16()
    C.gemm(big, big, torch.empty(4096, 4096, device="cuda", dtype=torch.bfloat16), config=0)
    test_linear_cross_entropy_gradients_with_few_rows(monkeypatch, rows, V, K, sparse)


@pytest.mark.parametrize("M,N,K,counts", [(256, 512, 32000, None), (300, 136, 20000, None), (513, 768, 30522, None), (1, 8, 50257, None), (2048, 264, 18440, None),
                                          (1500, 768, 30522, (0, 1, 255, 256, 257, 600, 1500)), (4096, 136, 8200, (1, 256, 2500, 4096)), (6000, 512, 32000, (37, 6000))])
def test_product_in_parts(C, M, N, K, counts):
    """dX = alpha dY W with its reduction in parts of a number that, with `counts`, only the device knows: ragged sizes, rows that take no part, memory that
    held NaN before. One rounding to bf16 (2^-8) of fp32 sums of exact products; the same bits again."""
    torch.manual_seed(N)
    dy = (torch.randn(M, (K + 7) // 8 * 8, device="cuda") * 0.1).bfloat16()[:, :K]
    w, alpha = torch.randn(K, N, device="cuda").bfloat16(), torch.tensor([-3.0], device="cuda")
    lin, size = -3.0 * (dy.double() @ w.double()), 3.0 * (dy.double().abs() @ w.double().abs())

    def run(*rows):
        torch.full((80 * 256 * 256,), float("nan"), device="cuda")     # freed: the scratch may take its place
        dx = torch.full((M, N), 7.0, device="cuda", dtype=torch.bfloat16)
        assert C.gemm_in_parts(dy, w, dx, alpha, *rows)
        assert C.read_status(0) == 0
        return dx

    C.clear_status(0)
    for m in counts or (None,):
        idx = torch.randperm(M, device="cuda")[:M].int()
        rows = () if m is None else (idx, torch.tensor([m, M], device="cuda", dtype=torch.int32))
        dx, again = run(*rows), run(*rows)
        assert torch.equal(dx, again)
        to = torch.arange(M, device="cuda") if m is None else idx[:m].long()
        n = M if m is None else m
        assert ((dx[to].double() - lin[:n]).abs() <= lin[:n].abs() * 2.0 ** -8 + 2.0 ** -20 * (size[:n] + 8)).all()
        left = torch.ones(M, dtype=torch.bool, device="cuda")
        left[to] = False
        assert (dx[left] == 7).all()


def test_product_in_parts_is_left_where_one_serves_better(C):
    for M, N, K, counted in ((256, 512, 2056, False), (256, 512, 8200, False), (8192, 512, 32000, False), (24576, 768, 30522, True), (4096, 768, 1000, True)):
        dy, w = torch.zeros(M, (K + 7) // 8 * 8, device="cuda", dtype=torch.bfloat16)[:, :K], torch.zeros(K, N, device="cuda", dtype=torch.bfloat16)
        dx = torch.ones(M, N, device="cuda", dtype=torch.bfloat16)
        rows = (torch.arange(M, device="cuda").int(), torch.tensor([M, M], device="cuda", dtype=torch.int32)) if counted else ()
        assert not C.gemm_in_parts(dy, w, dx, torch.ones(1, device="cuda"), *rows) and (dx == 1).all()


@pytest.mark.parametrize("rows,V,K,sparse", [(256, 32000, 512, False), (4096, 30522, 768, True), (1024, 8200, 256, True)])
def test_linear_cross_entropy_gives_dx_the_same_bits_again(C, monkeypatch, rows, V, K, sparse):
    from flodl_b200 import ops
    from flodl_b200.ops import core
    monkeypatch.setitem(core._EAGER, "min_numel", 0)
    torch.manual_seed(K)
    x, w = torch.randn(rows, K, device="cuda").bfloat16(), (torch.randn(V, K, device="cuda") * 0.05).bfloat16()
    t = torch.randint(0, V, (rows,), device="cuda")
    if sparse:
        t[torch.rand(rows, device="cuda") < 0.85] = -100
    grads = []
    for _ in range(4):
        xg = x.clone().requires_grad_()
        ops.linear_cross_entropy(xg, w, None, t, -100, sparse).backward()
        grads.append(xg.grad)
    assert all(torch.equal(grads[0], g) for g in grads[1:])


def test_linear_gradients_in_one_launch_are_refused_where_they_do_not_fit(C):
    dy, w, x = (torch.randn(s, device="cuda").bfloat16() for s in ((2048, 1024), (1024, 1024), (2048, 1024)))
    dx, dw, db = torch.zeros_like(x), torch.zeros(1024, 1024, device="cuda"), torch.zeros(1028, device="cuda")
    assert not C.gemm_backward(dy, w, x, dx, dw, db[1:1025])                                        # sums go out sixteen bytes at a time
    assert not C.gemm_backward(dy, w, x, torch.zeros(2048, 1028, device="cuda", dtype=torch.bfloat16)[:, 4:], dw)
    assert not C.gemm_backward(dy[:64], w, x[:64], dx[:64], dw)                                     # too little work
    assert not dx.any() and not dw.any() and not db.any()


def test_gemm_fp32_out_accumulate_splitk_alpha(C):
    M, N, K = 256, 384, 1024
    torch.manual_seed(1)
    a = torch.randn(K, M, device="cuda").bfloat16()   # MN-major A: dW = dY^T X
    b = torch.randn(K, N, device="cuda").bfloat16()
    ref = a.float().t() @ b.float()
    base = torch.randn(M, N, device="cuda")
    out = base.clone()
    C.gemm(a, b, out, True, True, accumulate=True)
    assert (out - (base + ref)).abs().max().item() < 0.02 * ref.abs().max().item()
    out2 = base.clone()
    C.gemm(a, b, out2, True, True, accumulate=True, split_k=4)
    assert (out2 - (base + ref)).abs().max().item() < 0.02 * ref.abs().max().item()
    out4 = base.clone()
    C.gemm(a, b, out4, True, True, accumulate=True, split_k=2, config=4)     # 128x192 tiles, 128+64 epilogue split
    assert (out4 - (base + ref)).abs().max().item() < 0.02 * ref.abs().max().item()
    alpha = torch.tensor([0.25], device="cuda")
    out3 = torch.empty(M, N, device="cuda")
    C.gemm(a, b, out3, True, True, alpha=alpha)
    assert (out3 - 0.25 * ref).abs().max().item() < 0.02 * ref.abs().max().item()


@pytest.mark.parametrize("M,N,K,b_mn,epi", [(1, 768, 768, False, 0), (77, 768, 3072, False, 0), (77, 3072, 768, False, 1), (128, 64, 64, True, 0), (129, 68, 72, False, 3),
                                            (300, 128, 520, True, 2), (512, 512, 128, True, 4), (130, 60, 4096, False, 0)])
def test_gemm_few_tiles(C, M, N, K, b_mn, epi, pad=4):
    """Products of few output tiles, which the dispatch gives to the kernel that splits K over a cluster: edges of tiles and of the split, both
    layouts of B, every epilogue, strided output. Against 64 bits: the output carries one rounding to bf16 (2^-8 at most), GELU' is taken of a
    stored, rounded value, the fast GELU adds 6e-5 absolute; in norm all of it stays below one such rounding."""
    torch.manual_seed(15)
    a = torch.randn(M, K + 8, device="cuda").bfloat16()[:, :K]
    b = (torch.randn(N, K, device="cuda") / math.sqrt(K)).bfloat16()
    bm = b.t().contiguous() if b_mn else b
    bias = torch.randn(N, device="cuda") if epi in (0, 1, 3) else None
    out = torch.zeros(M, N + pad, device="cuda").bfloat16()
    aux = torch.randn(M, N, device="cuda").bfloat16()
    alpha = torch.tensor([0.5], device="cuda") if epi == 0 else None
    C.clear_status(0)
    C.gemm(a, bm, out[:, :N], False, b_mn, bias=bias, epi=epi, aux=aux if epi else None, alpha=alpha)
    torch.cuda.synchronize()
    assert C.read_status(0) == 0
    pre = a.double() @ b.double().t() * (0.5 if epi == 0 else 1.0) + (0 if bias is None else bias.double())
    gelu = lambda x: torch.nn.functional.gelu(x, approximate="tanh" if epi > 2 else "none")
    if epi in (0, 1, 3):
        ref = pre if epi == 0 else gelu(pre)
        if epi:
            assert ((aux.double() - pre).norm() / pre.norm()).item() < 2 ** -8
    else:
        x = aux.double().requires_grad_(True)
        gelu(x).backward(pre)
        ref = x.grad
    assert ((out[:, :N].double() - ref).norm() / ref.norm()).item() < 2 ** -8
    assert torch.all(out[:, N:] == 0)


def _launched(call):
    """Names of the kernels that a call launches."""
    from torch.profiler import ProfilerActivity, profile
    call()
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CUDA]) as seen:
        call()
        torch.cuda.synchronize()
    return " ".join(e.name for e in seen.events() if e.device_type == torch.autograd.DeviceType.CUDA)


@pytest.mark.parametrize("M,N,K,kernel", [(96, 128, 64, "small"), (97, 128, 448, "bf16"), (97, 128, 512, "small"), (128, 37 * 64, 512, "small"), (128, 38 * 64, 512, "bf16"),
                                          (128, 74 * 64, 768, "small"), (128, 75 * 64, 768, "bf16"), (130, 64, 4096, "small"), (1, 768, 768, "small"),
                                          (2048, 1024, 1280, "split"), (2048, 1024, 1272, "bf16"), (1300, 504, 1544, "split"), (1800, 1000, 1352, "split"), (4096, 512, 2048, "split"),
                                          (4096, 3072, 2048, "bf16")])
@pytest.mark.parametrize("b_mn", [False, True])
def test_gemm_goes_to_the_kernel_that_the_dispatch_means(C, M, N, K, kernel, b_mn):
    """Both sides of each line of the dispatch, as it lies on 148 SMs, most shapes of the two tests around this one among them."""
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the lines are proportional to the number of SMs")
    a = torch.randn(M, K, device="cuda").bfloat16()
    b = torch.randn(*((K, N) if b_mn else (N, K)), device="cuda").bfloat16()
    out = torch.empty(M, N, device="cuda", dtype=torch.bfloat16)
    names = _launched(lambda: C.gemm(a, b, out, False, b_mn))
    assert f"gemm_{kernel}_kernel" in names, names
    A, B = a.double(), (b.t() if b_mn else b).double()
    ref = A @ B.t()
    assert ((out.double() - ref).norm() / ref.norm()).item() < 2 ** -8


@pytest.mark.parametrize("M,N,K,launches", [(512, 256, 256, 1), (200, 512, 512, 1), (128, 1536, 64, 1), (128, 1600, 64, 3)])
def test_grouped_gemm_is_one_launch_where_it_is_small(C, M, N, K, launches):
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the line is proportional to the number of SMs")
    a = torch.randn(M, K, device="cuda").bfloat16()
    ws = [(torch.randn(N, K, device="cuda") / math.sqrt(K)).bfloat16() for _ in range(3)]
    bs = [torch.randn(N, device="cuda") for _ in range(3)]
    out = torch.empty(M, 3 * N, device="cuda", dtype=torch.bfloat16)
    names = _launched(lambda: C.gemm_grouped(a, ws, out, bs))
    assert names.count("gemm_") == launches and (launches == 3 or "gemm_small_kernel" in names), names
    for g in range(3):
        ref = a.double() @ ws[g].double().t() + bs[g].double()
        assert ((out[:, g * N:(g + 1) * N].double() - ref).norm() / ref.norm()).item() < 2 ** -8


@pytest.mark.parametrize("M,N,K", [(1800, 1000, 1352), (1300, 504, 1544), (4096, 512, 2048)])
@pytest.mark.parametrize("b_mn", [False, True])
@pytest.mark.parametrize("epi", [0, 1, 2, 3, 4])
def test_gemm_two_pairs(C, M, N, K, b_mn, epi):
    """Products of 12 to 32 tiles of 256 x 256 and a long reduction, which the dispatch splits over two pairs of a cluster where the device holds
    that many clusters: whole and ragged tiles, an odd number of reduction steps. Bounds as for the products of few tiles."""
    test_gemm_few_tiles(C, M, N, K, b_mn, epi, pad=8)


@pytest.mark.parametrize("M,N,K", [(1800, 1000, 1352), (4096, 512, 2048)])
@pytest.mark.parametrize("pad,at", [(1, 0), (4, 0), (8, 1), (8, 4)])
def test_gemm_two_pairs_takes_pre_activations_at_any_alignment(C, M, N, K, pad, at):
    """GELU' over two pairs of a cluster where rows of the pre-activations are off a 16-byte boundary. Bounds as above."""
    torch.manual_seed(16)
    a, b = torch.randn(M, K, device="cuda").bfloat16(), (torch.randn(K, N, device="cuda") / math.sqrt(K)).bfloat16()
    aux = torch.randn(M, N + pad, device="cuda").bfloat16()[:, at:at + N]
    out = torch.zeros(M, N, device="cuda").bfloat16()
    for epi, approximate in ((2, "none"), (4, "tanh")):
        C.clear_status(0)
        C.gemm(a, b, out, False, True, epi=epi, aux=aux)
        assert C.read_status(0) == 0
        x = aux.double().requires_grad_(True)
        torch.nn.functional.gelu(x, approximate=approximate).backward(a.double() @ b.double())
        assert ((out.double() - x.grad).norm() / x.grad.norm()).item() < 2 ** -8


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("cols", [768, 512, 16 * 8, 1024])
def test_layernorm_fwd_bwd(C, dtype, cols):
    rows = 1000
    torch.manual_seed(2)
    x = torch.randn(rows, cols, device="cuda").to(dtype)
    r = torch.randn(rows, cols, device="cuda").to(dtype)
    g = torch.randn(cols, device="cuda")
    b = torch.randn(cols, device="cuda")
    y, pre, mean, rstd = C.layernorm_fwd(x, r, g, b, 1e-5, 0.0, 0, True)
    pre_ref = (x.float() + r.float()).to(dtype).float()
    ref = torch.nn.functional.layer_norm(pre_ref, (cols,), g, b, 1e-5)
    tol = 0.02 * ref.abs().max().item() if dtype == torch.bfloat16 else 1e-4
    assert (y.float() - ref).abs().max().item() < tol
    assert (pre.float() - pre_ref).abs().max().item() < 1e-6
    dy = torch.randn(rows, cols, device="cuda").to(dtype)
    dpre, _, dg, db = C.layernorm_bwd(dy, pre, mean, rstd, g, 0.0, 0, False, True, None, None)
    xr = pre_ref.clone().requires_grad_(True)
    gr = g.clone().requires_grad_(True)
    br = b.clone().requires_grad_(True)
    torch.nn.functional.layer_norm(xr, (cols,), gr, br, 1e-5).backward(dy.float())
    assert (dpre.float() - xr.grad).abs().max().item() < (0.02 * xr.grad.abs().max().item() + 0.02 if dtype == torch.bfloat16 else 1e-3)
    assert (dg - gr.grad).abs().max().item() < 5e-2 * max(1.0, gr.grad.abs().max().item()) * (1 if dtype == torch.bfloat16 else 0.01)
    assert (db - br.grad).abs().max().item() < 1e-2 * max(1.0, br.grad.abs().max().item())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("rows,cols", [(1, 256), (3, 264), (5000, 768), (4099, 1016), (20001, 320)])
def test_layernorm_rows_per_warp(C, dtype, rows, cols):
    """From fewer rows than warps to several rows per warp, columns that leave lanes idle; parameter gradients written and accumulated.
    Element-wise results carry one rounding to their type (2^-8 for bf16); the parameter gradients are 32-bit sums over the stored `pre`."""
    torch.manual_seed(14)
    x, r, dy = (torch.randn(rows, cols, device="cuda").to(dtype) for _ in range(3))
    g, b = torch.randn(cols, device="cuda"), torch.randn(cols, device="cuda")
    y, pre, mean, rstd = C.layernorm_fwd(x, r, g, b, 1e-5, 0.0, 0, True)
    leaves = [pre.double().requires_grad_(True), g.double().requires_grad_(True), b.double().requires_grad_(True)]
    ref = torch.nn.functional.layer_norm(leaves[0], (cols,), leaves[1], leaves[2], 1e-5)
    ref.backward(dy.double())
    unit = 2 ** -8 if dtype == torch.bfloat16 else 2 ** -18
    close = lambda got, want, u: ((got.double() - want).norm() / want.norm().clamp_min(1e-30)).item() < u
    # y, mean and rstd are made from the unrounded sum, the reference from the stored one: another rounding
    assert close(y, ref.detach(), 2 * unit)
    dpre, _, dg, db = C.layernorm_bwd(dy, pre, mean, rstd, g, 0.0, 0, False, True, None, None)
    acc_g, acc_b = torch.ones(cols + 1, device="cuda")[1:], torch.ones(cols, device="cuda")      # one off a 16-byte boundary
    dpre2, _, _, _ = C.layernorm_bwd(dy, pre, mean, rstd, g, 0.0, 0, False, True, acc_g, acc_b)
    assert torch.equal(dpre, dpre2) and close(dpre, leaves[0].grad, 2 * unit)
    assert close(dg, leaves[1].grad, 2 * unit)
    assert close(db, leaves[2].grad, 2 ** -18)
    assert close(acc_g - 1, dg.double(), 2 ** -14) and close(acc_b - 1, db.double(), 2 ** -14)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("rows,cols", [(1183, 128), (1185, 64), (2371, 256), (9473, 128), (3555, 768)])
def test_layernorm_backward_grids(C, dtype, rows, cols):
    """Row counts around those at which the backward pass takes fewer blocks than a wave; bounds as above."""
    test_layernorm_rows_per_warp(C, dtype, rows, cols)


@pytest.mark.parametrize("dtype,cols", [(torch.bfloat16, 768), (torch.bfloat16, 264), (torch.float32, 1024), (torch.float32, 36)])
@pytest.mark.parametrize("param", [torch.float32, torch.bfloat16])
def test_layernorm_parameters_around_few_rows(C, dtype, cols, param):
    """Either side of the row count (eight to an SM) up to which the parameters are loaded with the row; parameters of both types, on and off the
    alignment of a vector, and absent. 32-bit arithmetic, one rounding to the type of the result."""
    torch.manual_seed(15)
    few = 8 * torch.cuda.get_device_properties(0).multi_processor_count
    hold = torch.randn(2, cols + 1, device="cuda").to(param)
    for rows in (1, few, few + 1):
        x = torch.randn(rows, cols, device="cuda").to(dtype)
        for g, b in ((hold[0, :cols].clone(), hold[1, :cols].clone()), (hold[0, 1:], hold[1, 1:].clone()), (hold[0, :cols].clone(), hold[1, 1:]), (None, None)):
            y = C.layernorm_fwd(x, None, g, b, 1e-5, 0.0, 0, False)[0]
            ref = torch.nn.functional.layer_norm(x.double(), (cols,), None if g is None else g.double(), None if b is None else b.double(), 1e-5)
            assert ((y.double() - ref).norm() / ref.norm()).item() < (2 ** -8 if dtype == torch.bfloat16 else 2 ** -18)


@pytest.mark.parametrize("dtype,V", [(torch.bfloat16, 4104), (torch.bfloat16, 32768), (torch.bfloat16, 32776), (torch.float32, 16384), (torch.float32, 16388)])
def test_softmax_ce_block_sizes(C, dtype, V):
    """Either side of the row length at which a block's size changes, with more rows than resident blocks. The gradient carries one rounding to its
    type; the loss is a mean of 32-bit values near 10, each within two units in the last place."""
    torch.manual_seed(18)
    rows = 900
    x = torch.randn(rows, V, device="cuda").to(dtype)
    t = torch.randint(0, V, (rows,), device="cuda")
    loss, dl, _ = C.softmax_ce(x, t, -100, True, False)
    xd = x.double()
    p = torch.softmax(xd, 1)
    p[torch.arange(rows, device="cuda"), t] -= 1
    ref = torch.nn.functional.cross_entropy(xd, t)
    assert abs(loss.double().item() - ref.item()) < 2 ** -21 * abs(ref.item())
    assert ((dl.double() - p / rows).norm() / (p / rows).norm()).item() < (2 ** -8 if dtype == torch.bfloat16 else 2 ** -18)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("tokens,dim,ids", [(1, 8, "random"), (4099, 768, "equal"), (777, 1028, "runs"), (5000, 64, "random"), (33, 30, "runs")])
def test_embedding_bwd_runs(C, dtype, tokens, dim, ids):
    """Equal neighbours are summed in registers first; padding and a table row that nothing touches. Sums of 32 bits in any order."""
    torch.manual_seed(17)
    vocab = 50
    t = {"random": torch.randint(0, vocab - 1, (tokens,)), "equal": torch.full((tokens,), 7), "runs": (torch.arange(tokens) // 5) % (vocab - 1)}[ids].cuda()
    dy = torch.randn(tokens, dim, device="cuda").to(dtype)
    dw = torch.ones(vocab, dim, device="cuda")
    C.embedding_bwd(dy, t, dw, 3)
    ref = torch.ones(vocab, dim, device="cuda", dtype=torch.double).index_add_(0, t[t != 3], dy.double()[t != 3])
    assert ((dw.double() - ref).norm() / ref.norm()).item() < 2 ** -18 and torch.all(dw[vocab - 1] == 1)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("tokens", [1023, 1025, 8191, 8193, 16383, 16387])
def test_embedding_bwd_run_lengths(C, dtype, tokens):
    """Either side of the token counts at which a block's run of tokens and the rows in flight change; ids that repeat after 1 to 40 tokens."""
    torch.manual_seed(24)
    vocab, dim = 300, 36
    t = torch.repeat_interleave(torch.randint(0, vocab, (tokens,)), torch.randint(1, 41, (tokens,)))[:tokens].cuda()
    dy = torch.randn(tokens, dim, device="cuda").to(dtype)
    dw = torch.zeros(vocab, dim, device="cuda")
    C.embedding_bwd(dy, t, dw, 5)
    ref = torch.zeros(vocab, dim, device="cuda", dtype=torch.double).index_add_(0, t[t != 5], dy.double()[t != 5])
    assert ((dw.double() - ref).norm() / ref.norm()).item() < 2 ** -18 and torch.all(dw[5] == 0)


def test_layernorm_dropout_mask_consistent(C):
    rows, cols, p = 512, 768, 0.1
    x = torch.ones(rows, cols, device="cuda", dtype=torch.bfloat16)
    r = torch.zeros_like(x)
    _, pre, mean, rstd = C.layernorm_fwd(x, r, None, None, 1e-5, p, 1234, True)
    keep = (pre.float() != 0)
    frac = keep.float().mean().item()
    assert abs(frac - (1 - p)) < 0.01
    assert torch.allclose(pre.float()[keep], torch.full_like(pre.float()[keep], 1 / (1 - p)), atol=1e-2)
    # the standalone dropout kernel and the LN backward regenerate the same mask
    d = C.dropout(x, p, 1234)
    assert torch.equal(d.float() != 0, keep)
    dy = torch.ones_like(x)
    dpre, dxd, _, _ = C.layernorm_bwd(dy, pre, mean, rstd, None, p, 1234, True, False, None, None)
    assert ((dxd.float() != 0) & ~keep).sum().item() == 0


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("tanh", [False, True])
def test_gelu(C, dtype, tanh):
    x = torch.randn(4099 * 3, device="cuda").to(dtype)
    y = C.gelu_fwd(x, tanh)
    xr = x.float().requires_grad_(True)
    ref = torch.nn.functional.gelu(xr, approximate="tanh" if tanh else "none")
    tol = 0.02 if dtype == torch.bfloat16 else 1e-5
    assert (y.float() - ref).abs().max().item() < tol
    dy = torch.randn_like(x)
    dx = C.gelu_bwd(dy, x, tanh)
    ref.backward(dy.float())
    assert (dx.float() - xr.grad).abs().max().item() < (0.03 if dtype == torch.bfloat16 else 1e-4)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("rows,V,pad", [(256, 30522, 6), (128, 10, 0), (64, 32000, 0)])
def test_softmax_ce(C, dtype, rows, V, pad):
    torch.manual_seed(3)
    buf = torch.randn(rows, V + pad, device="cuda").to(dtype) * 3
    logits = buf[:, :V]
    tgt = torch.randint(0, V, (rows,), device="cuda")
    tgt[::3] = -100
    lr = logits.float().clone().requires_grad_(True)
    ref = torch.nn.functional.cross_entropy(lr, tgt, ignore_index=-100)
    ref.backward()
    loss, dl, cinv = C.softmax_ce(logits, tgt, -100, True, False)
    assert abs(loss.item() - ref.item()) < (2e-2 if dtype == torch.bfloat16 else 1e-4)
    assert (dl.float() - lr.grad).abs().max().item() < (2e-3 if dtype == torch.bfloat16 else 1e-6)
    assert cinv[0].item() == (tgt != -100).sum().item()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("rows,V,offset", [(9, 1, 0), (33, 37, 0), (17, 2049, 1), (21, 4097, 3), (1000, 100, 0), (500, 30522, 0), (3, 50001, 1)])
def test_softmax_ce_row_alignments(C, dtype, rows, V, offset):
    """Contiguous rows of any length, i.e. of every alignment, starting off a 16-byte boundary too; some values -inf, as masks leave
    them; the gradient in a buffer of its own and in place. One rounding of the gradient to its type (2^-8 for bf16), whose largest value is
    1 / rows; sums in another order where the two buffers are aligned differently."""
    torch.manual_seed(13)
    flat = torch.randn(rows * V + offset, device="cuda").to(dtype) * 3
    logits = flat[offset:].view(rows, V)
    tgt = torch.randint(0, V, (rows,), device="cuda")
    if V > 8:
        logits[:, : V // 2] = float("-inf")
        tgt = tgt % (V - V // 2) + V // 2
    tgt[1::5] = -100
    lr = logits.double().requires_grad_(True)
    ref = torch.nn.functional.cross_entropy(lr, tgt, ignore_index=-100)
    ref.backward()
    n = int((tgt != -100).sum())
    tol = (2 ** -8 if dtype == torch.bfloat16 else 2 ** -20) / n
    loss, dl, _ = C.softmax_ce(logits, tgt, -100, True, False)
    assert abs(loss.item() - ref.item()) < 1e-5 * max(1.0, abs(ref.item()))
    assert (dl.double() - lr.grad).abs().max().item() <= tol
    scaled = dl.clone()
    C.scale_rows(scaled, torch.ones(1, device="cuda"))
    assert torch.equal(scaled, dl)
    C.scale_rows(scaled, torch.full((1,), 0.3, device="cuda"))
    assert (scaled.double() - 0.3 * dl.double()).abs().max().item() <= tol
    loss2, dl2, _ = C.softmax_ce(logits, tgt, -100, True, True)
    assert dl2.data_ptr() == logits.data_ptr() and (dl2.double() - lr.grad).abs().max().item() <= tol
    assert abs(loss2.item() - ref.item()) < 1e-5 * max(1.0, abs(ref.item()))


@pytest.mark.parametrize("dtype,V", [(torch.bfloat16, v) for v in (512, 513, 1024, 1025, 10240, 10241, 16384, 16385)] +
                         [(torch.float32, v) for v in (256, 257, 512, 513, 5120, 5121, 8192, 8193, 24576, 24577)])
@pytest.mark.parametrize("rows", [7, 601])
def test_softmax_ce_either_side_of_each_block_size(C, dtype, V, rows):
    """Row lengths at which the threads of a row change, of few rows and of many; bounds as above."""
    torch.manual_seed(23)
    x = torch.randn(rows, V, device="cuda").to(dtype)
    t = torch.randint(0, V, (rows,), device="cuda")
    t[::6] = -100
    n = int((t != -100).sum())
    xd = x.double()
    ref = torch.nn.functional.cross_entropy(xd, t, ignore_index=-100)
    p = torch.softmax(xd, 1)
    p[torch.arange(rows, device="cuda"), t.clamp_min(0)] -= 1
    p[t == -100] = 0
    for inplace in (False, True):
        loss, dl, _ = C.softmax_ce(x, t, -100, True, inplace)
        assert abs(loss.double().item() - ref.item()) < 2 ** -21 * abs(ref.item())
        assert ((dl.double() - p / n).norm() / (p / n).norm()).item() < (2 ** -8 if dtype == torch.bfloat16 else 2 ** -18)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("V", [1, 10, 4097])
def test_softmax_ce_nan_logit(C, dtype, V):
    """One NaN among a row's logits, wherever it is and also where a thread sees nothing else: the loss and that row's gradient are NaN, the other
    rows' gradients are not."""
    torch.manual_seed(22)
    rows = 9
    tgt = torch.randint(0, V, (rows,), device="cuda")
    for at in sorted({0, 1 % V, V // 2, V - 1}):
        x = torch.randn(rows, V, device="cuda").to(dtype)
        x[4, at] = float("nan")
        loss, dl, _ = C.softmax_ce(x, tgt, -100, True, False)
        assert torch.isnan(loss).item(), at
        nan = torch.isnan(dl.float())
        assert torch.all(nan[4]) and not torch.any(nan[:4]) and not torch.any(nan[5:]), at


def test_adam_matches_reference(C):
    n = 100003
    torch.manual_seed(4)
    p = torch.randn(n, device="cuda")
    g = torch.randn(n, device="cuda")
    m = torch.zeros(n, device="cuda")
    v = torch.zeros(n, device="cuda")
    p16 = torch.empty(n, device="cuda", dtype=torch.bfloat16)
    pr = p.clone()
    mr, vr = m.clone(), v.clone()
    lr, b1, b2, eps, wd = 1e-2, 0.9, 0.999, 1e-8, 0.01
    for t in range(1, 4):
        hyper = torch.tensor([lr, 1 - b1 ** t, 1 - b2 ** t, wd], device="cuda")
        C.adam_step(p, g, m, v, p16, hyper, b1, b2, eps)
        pr *= 1 - lr * wd
        mr = b1 * mr + (1 - b1) * g
        vr = b2 * vr + (1 - b2) * g * g
        pr -= (lr / (1 - b1 ** t)) * mr / ((vr / (1 - b2 ** t)).sqrt() + eps)
    assert (p - pr).abs().max().item() < 1e-5
    assert (p16.float() - pr).abs().max().item() < 2e-2
    # bf16 gradients + device-side gradient scale
    gs = torch.tensor([0.5], device="cuda")
    p2, m2, v2 = pr.clone(), torch.zeros(n, device="cuda"), torch.zeros(n, device="cuda")
    hyper = torch.tensor([lr, 1 - b1, 1 - b2, 0.0], device="cuda")
    C.adam_step(p2, g.bfloat16(), m2, v2, None, hyper, b1, b2, eps, gs)
    gq = g.bfloat16().float() * 0.5
    ref = pr - (lr / (1 - b1)) * ((1 - b1) * gq) / ((((1 - b2) * gq * gq) / (1 - b2)).sqrt() + eps)
    assert (p2 - ref).abs().max().item() < 1e-5


def test_sgd_matches_reference(C):
    n = 5001
    p = torch.randn(n, device="cuda")
    g = torch.randn(n, device="cuda")
    buf = torch.zeros(n, device="cuda")
    pr, br = p.clone(), None
    lr, mu, wd = 0.1, 0.9, 1e-4
    for step in range(3):
        hyper = torch.tensor([lr, mu, wd, 1.0 if step == 0 else 0.0], device="cuda")
        C.sgd_step(p, g, buf, None, hyper)
        gg = g + wd * pr
        br = gg.clone() if br is None else mu * br + gg
        pr = pr - lr * br
    assert (p - pr).abs().max().item() < 1e-5


def test_grad_norm_and_clip(C):
    g = torch.randn(1_000_003, device="cuda")
    out = C.grad_norm(g, 1.0, 1.0)
    ref = g.double().norm().item()
    assert abs(out[0].item() - ref) / ref < 1e-5
    assert abs(out[1].item() - 1.0 / (ref + 1e-6)) < 1e-6
    out = C.grad_norm(g.bfloat16(), 0.0, 1.0)
    assert abs(out[0].item() - g.bfloat16().double().norm().item()) / ref < 1e-4
    assert out[1].item() == 1.0


def test_colsum_and_cast(C):
    x = torch.randn(4096, 770, device="cuda").bfloat16()
    out = torch.zeros(770, device="cuda")
    C.colsum(x, out)
    assert (out - x.float().sum(0)).abs().max().item() < 1e-2
    y = torch.empty(4096 * 770, device="cuda")
    C.cast_into(x.view(-1), y, 2.0)
    assert torch.equal(y, x.view(-1).float() * 2)


def _attn_ref(q, k, v, mask, scale, causal):
    # q, k, v: [B, S, H, D] fp32
    qh, kh, vh = (t.permute(0, 2, 1, 3) for t in (q, k, v))
    s = (qh @ kh.transpose(-1, -2)) * scale
    if mask is not None:
        s = s + mask[:, None, None, :]
    if causal:
        S = q.shape[1]
        s = s.masked_fill(torch.ones(S, S, device=q.device).triu(1).bool(), float("-inf"))
    p = torch.softmax(s, dim=-1)
    return (p @ vh).permute(0, 2, 1, 3)


@pytest.mark.parametrize("B,H,S,causal,use_mask", [(2, 3, 128, False, True), (2, 2, 256, True, False), (1, 2, 256, False, True), (2, 2, 384, True, False), (1, 1, 200, False, False),
                                                        # one key block: the kernels that share an SM between four / two CTAs
                                                        (4, 12, 128, True, False), (3, 2, 77, False, True), (2, 4, 64, True, False), (32, 12, 128, False, True)])
def test_attention_fwd_bwd(C, B, H, S, causal, use_mask):
    torch.manual_seed(5)
    D = 64
    qkv = torch.randn(B, S, 3, H, D, device="cuda").bfloat16()
    q, k, v = qkv[:, :, 0], qkv[:, :, 1], qkv[:, :, 2]
    mask = None
    if use_mask:
        mask = torch.zeros(B, S, device="cuda")
        mask[:, S - 17:] = -1e4
    scale = 1.0 / math.sqrt(D)
    C.clear_status(0)
    o, lse = C.attn_fwd(q, k, v, mask, scale, causal)
    torch.cuda.synchronize()
    assert C.read_status(0) == 0
    qf, kf, vf = (t.float().clone().requires_grad_(True) for t in (q, k, v))
    ref = _attn_ref(qf, kf, vf, mask, scale, causal)
    assert (o.float() - ref).abs().max().item() < 0.03, (o.float() - ref).abs().max().item()
    do = torch.randn(B, S, H, D, device="cuda").bfloat16()
    dqkv = C.attn_bwd(q, k, v, o, do, lse, mask, scale, causal)
    torch.cuda.synchronize()
    assert C.read_status(0) == 0
    ref.backward(do.float())
    for i, g in enumerate((qf.grad, kf.grad, vf.grad)):
        err = (dqkv[:, :, i].float() - g).abs().max().item()
        assert err < 0.06 * max(1.0, g.abs().max().item()), (i, err, g.abs().max().item())


@pytest.mark.parametrize("S", [18, 32, 33, 64, 65, 96, 97])
def test_attention_up_to_the_end_of_a_short_sequence(C, S):
    """Either side of the lengths at which thirty-two keys more are worked on; bounds as above."""
    for causal, use_mask in ((False, True), (True, False)):
        test_attention_fwd_bwd(C, 2, 3, S, causal, use_mask)


@pytest.mark.parametrize("B,H,S,causal,use_mask", [(1, 1, 129, True, False), (2, 3, 131, False, True), (1, 2, 255, True, True), (3, 1, 257, False, False),
                                                   (1, 4, 509, False, True), (2, 2, 641, True, False), (9, 20, 129, False, False), (1, 1, 2050, True, False)])
def test_attention_several_key_blocks(C, B, H, S, causal, use_mask):
    """Sizes at the edges of the 128-row blocks, against 64-bit attention. Inputs and outputs are rounded to bf16 (2^-9 relative each), and so
    are the probabilities and their gradients inside; four such roundings in root-sum-square are 2^-8 of a result's norm."""
    torch.manual_seed(11)
    qkv = torch.randn(B, S, 3, H, 64, device="cuda").bfloat16()
    q, k, v = qkv[:, :, 0], qkv[:, :, 1], qkv[:, :, 2]
    mask = None
    if use_mask:
        mask = torch.zeros(B, S, device="cuda")
        mask[:, S // 3:] = -1e4
        mask[0] = 0.0
    C.clear_status(0)
    o, lse = C.attn_fwd(q, k, v, mask, 0.125, causal)
    do = torch.randn(B, S, H, 64, device="cuda").bfloat16()
    dqkv = C.attn_bwd(q, k, v, o, do, lse, mask, 0.125, causal)
    torch.cuda.synchronize()
    assert C.read_status(0) == 0
    ref_in = [t.double().requires_grad_(True) for t in (q, k, v)]
    ref = _attn_ref(*ref_in, None if mask is None else mask.double(), 0.125, causal)
    ref.backward(do.double())
    assert ((o.double() - ref).norm() / ref.norm()).item() < 2 ** -8
    for i, t in enumerate(ref_in):
        assert ((dqkv[:, :, i].double() - t.grad).norm() / t.grad.norm()).item() < 2 ** -7, i     # through P and dS both


def test_attention_running_maximum(C):
    """A key of a later block outweighs the first block's by a factor of 2^1 to 2^8, and it alone has a value: the output is that value over the
    row's 32-bit sum. Relative to the row's true maximum its probability is 1, so that only the output's own rounding to bf16 is left: 2^-8 of each
    value at most, and 2^-6 of that for the 32-bit sums and exponentials."""
    S, D = 384, 64
    torch.manual_seed(19)
    qkv = torch.zeros(1, S, 3, 1, D, device="cuda").bfloat16()
    q, k, v = qkv[:, :, 0], qkv[:, :, 1], qkv[:, :, 2]
    q[0, :, 0, 0] = torch.linspace(0.7, 5.5, S, device="cuda").bfloat16()       # the key's score above the others', in natural units
    k[0, 200, 0, 0] = 8.0
    v[0, 200, 0] = torch.randn(D, device="cuda").bfloat16()
    o, lse = C.attn_fwd(q, k, v, None, 0.125, False)
    ref = _attn_ref(q.double(), k.double(), v.double(), None, 0.125, False)
    assert ((o.double() - ref).abs() / ref.abs()).max().item() < 2 ** -8 * (1 + 2 ** -6)
    x = q[0, :, 0, 0].double()
    assert (lse[0, 0].double() - torch.log(x.exp() + S - 1)).abs().max().item() < 2 ** -18


def test_attention_mask_common_to_all_keys(C):
    """A mask value that all keys of a text share does not change the softmax. The score plus -1e6 keeps three bits after the point in
    32 bits; the kernel has to take the maximum off the mask before it adds the score. Bound as for the cases above: 2^-8 in norm."""
    torch.manual_seed(20)
    for S, causal in ((300, False), (300, True), (640, False)):
        q, k, v = torch.randn(2, S, 3, 2, 64, device="cuda").bfloat16().unbind(2)
        mask = torch.zeros(2, S, device="cuda")
        mask[1] = -1e6
        o, _ = C.attn_fwd(q, k, v, mask, 0.125, causal)
        ref = _attn_ref(q.double(), k.double(), v.double(), None, 0.125, causal)
        for b in range(2):
            assert ((o[b].double() - ref[b]).norm() / ref[b].norm()).item() < 2 ** -8, (S, causal, b)


@pytest.mark.parametrize("B,H,S,causal", [(4, 12, 384, False), (2, 5, 385, False), (3, 7, 1000, False), (8, 12, 1024, True), (1, 30, 1333, True)])
def test_attention_backward_repeats_itself(C, B, H, S, causal):
    """dQ is a sum over the CTAs of a head, added in a fixed order: the same bits from every call."""
    torch.manual_seed(21)
    q, k, v = torch.randn(B, S, 3, H, 64, device="cuda").bfloat16().unbind(2)
    o, lse = C.attn_fwd(q, k, v, None, 0.125, causal)
    do = torch.randn_like(o)
    C.clear_status(0)
    first = C.attn_bwd(q, k, v, o, do, lse, None, 0.125, causal)
    for _ in range(5):
        assert torch.equal(C.attn_bwd(q, k, v, o, do, lse, None, 0.125, causal), first)
    assert C.read_status(0) == 0


def test_attention_several_key_blocks_dropout(C):
    """O is linear in V for fixed probabilities, so <dO, O> = <dV, V> exactly if and only if backward drops what forward dropped."""
    torch.manual_seed(12)
    qkv = torch.randn(2, 300, 3, 2, 64, device="cuda").bfloat16()
    q, k, v = qkv[:, :, 0], qkv[:, :, 1], qkv[:, :, 2]
    o, lse = C.attn_fwd(q, k, v, None, 0.125, False, 0.25, 77)
    do = o.detach().clone()             # every term of <dO, O> positive: no cancellation, a relative bound of two roundings holds
    dqkv = C.attn_bwd(q, k, v, o, do, lse, None, 0.125, False, 0.25, 77)
    a, b = (do.double() * o.double()).sum().item(), (dqkv[:, :, 2].double() * v.double()).sum().item()
    assert abs(a - b) < 2 ** -7 * abs(a), (a, b)


def _attn_restated(q, k, v, do, mask, scale, causal, z=None):
    """Output and gradients of attention in 64 bits, exact, and again with what the kernels round to bf16 rounded: O before it is used in D, the
    probabilities and dS before their products. A row without a live key has an output and gradients of zero."""
    q, k, v, do = (t.double().permute(0, 2, 1, 3) for t in (q, k, v, do))
    s = q @ k.transpose(-1, -2) * scale
    if mask is not None:
        s = s + mask.double()[:, None, None, :]
    if causal:
        s = s.masked_fill(torch.ones(s.shape[-2:], dtype=torch.bool, device=s.device).triu(1), float("-inf"))
    p = torch.softmax(s, -1).nan_to_num(0.0)
    z = torch.ones_like(p) if z is None else z

    def results(r):
        o = (r(p * z) @ v)
        ds = r(p * (do @ v.transpose(-1, -2) * z - (do * r(o)).sum(-1, keepdim=True)) * scale)
        return [t.permute(0, 2, 1, 3) for t in (o, ds @ k, ds.transpose(-1, -2) @ q, r(p * z).transpose(-1, -2) @ do)]

    return results(lambda t: t), results(lambda t: t.bfloat16().double())


def _attn_check(C, q, k, v, mask, scale, causal, p_drop=0.0, seed=0, z=None):
    """Forward and backward against 64 bits: in norm at most twice as far off as the restatement that rounds where the kernels have to, and the
    rounding of the results themselves (2^-9)."""
    do = torch.randn_like(q).contiguous()
    C.clear_status(0)
    o, lse = C.attn_fwd(q, k, v, mask, scale, causal, p_drop, seed)
    dqkv = C.attn_bwd(q, k, v, o, do, lse, mask, scale, causal, p_drop, seed)
    assert C.read_status(0) == 0
    exact, rounded = _attn_restated(q, k, v, do, mask, scale, causal, z)
    for name, got, want, near in zip(("o", "dq", "dk", "dv"), (o, dqkv[:, :, 0], dqkv[:, :, 1], dqkv[:, :, 2]), exact, rounded):
        assert torch.isfinite(got.float()).all(), name
        err, norm = (got.double() - want).norm().item(), want.norm().item()
        assert err <= 2 * (near - want).norm().item() + 2 ** -9 * norm + 1e-30, (name, err / norm, ((near - want).norm() / norm).item())
    return o, lse, dqkv


@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("scale", [0.125, -0.125])
@pytest.mark.parametrize("S", [257, 641])
def test_attention_growing_maxima(C, S, scale, causal):
    """Row maxima that grow by ten and more in log2 from block to block in every other row, and hardly in the rows between, so that the accumulator is
    rescaled in some rows of a warp; scores of either sign of the scale."""
    torch.manual_seed(25)
    q, k, v = (t.clone() for t in torch.randn(2, S, 3, 2, 64, device="cuda").bfloat16().unbind(2))       # three tensors, not slices of one
    q[:, 1::2] *= 0.05
    k *= (1 + 3 * (torch.arange(S, device="cuda") // 128))[None, :, None, None]
    _attn_check(C, q, k, v, None, scale, causal)


@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("value", [-1e4, float("-inf")])
def test_attention_first_block_and_whole_texts_masked(C, value, causal):
    """Padding on the left that covers the first key block and more (the maximum starts at -inf, or far below), a text of which every key is masked, and
    one of which none is. Where -inf leaves a row no key at all, output and gradients are zero."""
    torch.manual_seed(26)
    B, S = 3, 400
    q, k, v = torch.randn(B, S, 3, 2, 64, device="cuda").bfloat16().unbind(2)
    mask = torch.zeros(B, S, device="cuda")
    mask[0, :150] = value
    mask[1] = value
    o, lse, dqkv = _attn_check(C, q, k, v, mask, 0.125, causal)
    if value == float("-inf"):
        dead = torch.zeros(B, S, dtype=torch.bool, device="cuda")
        dead[1] = True
        if causal:
            dead[0, :150] = True
        assert torch.all(o[dead] == 0) and torch.all(dqkv[:, :, 0][dead] == 0) and torch.all(lse.permute(0, 2, 1)[dead] == float("-inf"))
        assert torch.all(dqkv[1] == 0)


@pytest.mark.parametrize("causal,use_mask", [(False, False), (True, False), (False, True), (True, True)])
def test_attention_several_key_blocks_dropout_gradients(C, causal, use_mask):
    """All three gradients under dropout. The factors are read off the forward pass: with equal scores an output is the mean over the keys of factor times
    value, and values that are unit vectors for 64 keys at a time pick the factors out."""
    torch.manual_seed(27)
    B, S, H, p_drop, seed = 2, 300, 2, 0.25, 77
    zero = torch.zeros(B, S, H, 64, device="cuda").bfloat16()
    z = torch.empty(B, H, S, S, device="cuda", dtype=torch.double)
    for k0 in range(0, S, 64):
        n = min(64, S - k0)
        unit = zero.clone()
        unit[:, k0:k0 + n] = torch.eye(64, device="cuda")[:n, None].bfloat16()
        o, _ = C.attn_fwd(zero, zero, unit, None, 0.125, False, p_drop, seed)
        z[..., k0:k0 + n] = (o.double().permute(0, 2, 1, 3)[..., :n] > 0).double() / (1 - p_drop)
    assert abs((z > 0).double().mean().item() - (1 - p_drop)) < 0.01
    q, k, v = torch.randn(B, S, 3, H, 64, device="cuda").bfloat16().unbind(2)
    mask = None
    if use_mask:
        mask = torch.zeros(B, S, device="cuda")
        mask[0, 200:] = -1e4
    _attn_check(C, q, k, v, mask, 0.125, causal, p_drop, seed, z)


def test_attention_dropout_statistics(C):
    torch.manual_seed(6)
    B, H, S, D = 2, 2, 128, 64
    qkv = torch.zeros(B, S, 3, H, D, device="cuda").bfloat16()
    qkv[:, :, 2] = 1.0   # V = 1 -> each output = sum of kept probabilities / (1 - p)
    o, _ = C.attn_fwd(qkv[:, :, 0], qkv[:, :, 1], qkv[:, :, 2], None, 0.125, False, 0.25, 77)
    m = o.float().mean().item()
    assert abs(m - 1.0) < 0.02
    assert o.float().std().item() > 0.01


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("relu,use_res", [(False, False), (True, False), (True, True)])
@pytest.mark.parametrize("channels_last", [False, True])
def test_batchnorm_fused(C, dtype, relu, use_res, channels_last):
    torch.manual_seed(8)
    N, Ch, H = 16, 32, 8
    fmt = torch.channels_last if channels_last else torch.contiguous_format
    x = torch.randn(N, Ch, H, H, device="cuda").to(dtype).contiguous(memory_format=fmt)
    res = torch.randn(N, Ch, H, H, device="cuda").to(dtype).contiguous(memory_format=fmt) if use_res else None
    g = torch.rand(Ch, device="cuda") + 0.5
    b = torch.randn(Ch, device="cuda")
    rm, rv = torch.zeros(Ch, device="cuda"), torch.ones(Ch, device="cuda")
    rm_ref, rv_ref = rm.clone(), rv.clone()
    y, mean, rstd = C.bn_fwd(x, res, g, b, rm, rv, 1e-5, 0.1, relu, True)
    xr = x.float().clone().requires_grad_(True)
    gr, br = g.clone().requires_grad_(True), b.clone().requires_grad_(True)
    rr = res.float().clone().requires_grad_(True) if use_res else None
    ref = torch.nn.functional.batch_norm(xr, rm_ref, rv_ref, gr, br, True, 0.1, 1e-5)
    if use_res:
        ref = ref + rr
    if relu:
        ref = torch.relu(ref)
    tol = 0.05 if dtype == torch.bfloat16 else 1e-4
    assert (y.float() - ref).abs().max().item() < tol
    assert (rm - rm_ref).abs().max().item() < 1e-4 and (rv - rv_ref).abs().max().item() < 1e-3
    assert y.is_contiguous(memory_format=fmt)
    dy = torch.randn_like(ref).to(dtype).contiguous(memory_format=fmt)
    dx, dres, dg, db = C.bn_bwd(dy, x, y, g, mean, rstd, relu, use_res, None, None)
    # reference backward with the kernel's own ReLU mask (ties at 0 in bf16 would otherwise differ)
    (ref * (y.float() > 0 if relu else 1)).backward(dy.float()) if False else ref.backward(dy.float())
    btol = 0.08 if dtype == torch.bfloat16 else 2e-3
    assert (dx.float() - xr.grad).abs().max().item() < btol
    assert (dg - gr.grad).abs().max().item() < btol * 10 and (db - br.grad).abs().max().item() < btol * 10
    if use_res:
        assert (dres.float() - rr.grad).abs().max().item() < btol


def test_batchnorm_channels_last_many_blocks_accumulates(C):
    # enough pixels for several hundred blocks: exercises the last-block fold, the counter reset
    # (two calls in a row) and accumulation into existing gradient slots
    torch.manual_seed(9)
    x = torch.randn(64, 16, 32, 32, device="cuda").bfloat16().contiguous(memory_format=torch.channels_last)
    g, b = torch.rand(16, device="cuda") + 0.5, torch.randn(16, device="cuda")
    rm, rv = torch.zeros(16, device="cuda"), torch.ones(16, device="cuda")
    for _ in range(2):
        y, mean, rstd = C.bn_fwd(x, None, g, b, rm, rv, 1e-5, 0.1, False, True)
    ref = torch.nn.functional.batch_norm(x.float(), None, None, g, b, True, 0.1, 1e-5)
    assert (y.float() - ref).abs().max().item() < 0.05
    assert (mean - x.float().mean(dim=(0, 2, 3))).abs().max().item() < 1e-3
    dy = torch.randn_like(x)
    dg_acc, db_acc = torch.ones(16, device="cuda"), torch.ones(16, device="cuda")
    dx, _, _, _ = C.bn_bwd(dy, x, y, g, mean, rstd, False, False, dg_acc, db_acc)
    xr = x.float().clone().requires_grad_(True)
    gr, br = g.clone().requires_grad_(True), b.clone().requires_grad_(True)
    torch.nn.functional.batch_norm(xr, None, None, gr, br, True, 0.1, 1e-5).backward(dy.float())
    assert (dx.float() - xr.grad).abs().max().item() < 0.08
    assert (dg_acc - 1 - gr.grad).abs().max().item() < 0.02 * gr.grad.abs().max().item() + 0.5
    assert (db_acc - 1 - br.grad).abs().max().item() < 0.02 * br.grad.abs().max().item() + 0.5


@pytest.mark.parametrize("dtype,Ch", [(torch.float32, 4), (torch.bfloat16, 8), (torch.bfloat16, 24), (torch.bfloat16, 64), (torch.float32, 132), (torch.bfloat16, 136),
                                      (torch.float32, 256)])
@pytest.mark.parametrize("pixels", [37, 40000])
def test_batchnorm_channels_last_sums(C, dtype, Ch, pixels):
    """From one block to a full wave of them, channel counts that do and do not divide the block: the statistics and the parameter gradients
    are 32-bit sums over the stored values, whose error grows with the number of terms a thread adds (under a hundred here): 2^-17 in norm."""
    torch.manual_seed(16)
    x, dy = (torch.randn(1, Ch, pixels, 2, device="cuda").to(dtype).contiguous(memory_format=torch.channels_last) for _ in range(2))
    g, b = torch.rand(Ch, device="cuda") + 0.5, torch.randn(Ch, device="cuda")
    rm, rv = torch.zeros(Ch, device="cuda"), torch.ones(Ch, device="cuda")
    y, mean, rstd = C.bn_fwd(x, None, g, b, rm, rv, 1e-5, 0.1, False, True)
    xd, dyd = x.double(), dy.double()
    sd = (xd.var((0, 2, 3), unbiased=False) + 1e-5).rsqrt()
    close = lambda got, want: ((got.double() - want).norm() / want.norm()).item() < 2 ** -17
    assert (mean.double() - xd.mean((0, 2, 3))).abs().max().item() < 2 ** -17 and close(rstd, sd)
    _, _, dg, db = C.bn_bwd(dy, x, y, g, mean, rstd, False, False, None, None)
    xh = (xd - mean.double().view(-1, 1, 1)) * rstd.double().view(-1, 1, 1)
    assert close(dg, (dyd * xh).sum((0, 2, 3))) and close(db, dyd.sum((0, 2, 3)))


@pytest.mark.parametrize("N,Ci,Co,HW,k,stride", [(8, 16, 16, 32, 3, 1), (4, 16, 32, 32, 3, 2), (4, 32, 32, 16, 3, 1), (4, 32, 64, 16, 3, 2),
                                                 (6, 64, 64, 8, 3, 1), (4, 16, 32, 32, 1, 2), (2, 32, 8, 16, 3, 1), (150, 16, 16, 32, 3, 1), (2, 64, 16, 64, 3, 1), (3, 16, 32, 28, 3, 1), (2, 32, 64, 7, 3, 1), (300, 32, 32, 16, 3, 1)])
def test_conv_wgrad_tensor_core(C, N, Ci, Co, HW, k, stride):
    torch.manual_seed(11)
    pad = k // 2
    assert C.conv_wgrad_supported(N, HW, HW, Ci, Co, k, stride, pad)
    x = torch.randn(N, Ci, HW, HW, device="cuda").bfloat16().contiguous(memory_format=torch.channels_last)
    Ho = (HW + 2 * pad - k) // stride + 1
    dy = (torch.randn(N, Co, Ho, Ho, device="cuda") * 0.1).bfloat16().contiguous(memory_format=torch.channels_last)
    base = torch.randn(Co, Ci, k, k, device="cuda").contiguous(memory_format=torch.channels_last)
    dw = base.clone()
    assert dw.is_contiguous(memory_format=torch.channels_last)
    C.conv_wgrad(x, dy, dw, stride, pad)
    torch.cuda.synchronize()
    assert C.read_status(0) == 0
    ref = torch.nn.grad.conv2d_weight(x.float(), (Co, Ci, k, k), dy.float(), stride=stride, padding=pad)
    err = (dw - base - ref).abs().max().item()
    assert err <= 0.01 * ref.abs().max().item() + 0.02, f"max err {err} (ref max {ref.abs().max().item()})"
    # a second call accumulates again
    C.conv_wgrad(x, dy, dw, stride, pad)
    assert (dw - base - 2 * ref).abs().max().item() <= 0.02 * ref.abs().max().item() + 0.04


def test_conv_wgrad_rejects_unsupported(C):
    assert not C.conv_wgrad_supported(4, 32, 32, 3, 16, 3, 1, 1)       # 3 input channels: rows are not 16-byte multiples
    assert not C.conv_wgrad_supported(4, 32, 32, 16, 16, 5, 1, 2)      # 5x5
    assert not C.conv_wgrad_supported(4, 28, 28, 16, 16, 3, 2, 1)      # strided, width not a power of two


@pytest.mark.parametrize("N,Ci,Co,HW,k,stride", [(8, 16, 16, 32, 3, 1), (4, 16, 32, 32, 3, 2), (4, 32, 32, 16, 3, 1), (4, 32, 64, 16, 3, 2),
                                                 (5, 64, 64, 8, 3, 1), (4, 16, 32, 32, 1, 2), (2, 32, 16, 16, 3, 1), (160, 16, 16, 32, 3, 1),
                                                 (2, 64, 48, 64, 3, 1), (3, 16, 32, 28, 3, 1), (2, 32, 32, 7, 3, 1), (12, 64, 64, 64, 3, 1)])
def test_conv_fprop_tensor_core(C, N, Ci, Co, HW, k, stride):
    torch.manual_seed(12)
    pad = k // 2
    assert C.conv_fprop_supported(N, HW, HW, Ci, Co, k, stride, pad)
    x = torch.randn(N, Ci, HW, HW, device="cuda").bfloat16().contiguous(memory_format=torch.channels_last)
    w = (torch.randn(Co, Ci, k, k, device="cuda") * 0.1).bfloat16().contiguous(memory_format=torch.channels_last)
    stats = torch.zeros(2, Co, device="cuda")
    y = C.conv_fprop(x, w, stride, pad, stats)
    torch.cuda.synchronize()
    assert C.read_status(0) == 0
    ref = F.conv2d(x.float(), w.float(), None, stride, pad)
    assert y.shape == ref.shape and y.is_contiguous(memory_format=torch.channels_last)
    err = (y.float() - ref).abs().max().item()
    assert err <= 0.01 * ref.abs().max().item() + 0.01, f"max err {err} (ref max {ref.abs().max().item()})"
    # the fused statistics are those of the rounded output
    yf = y.float()
    s1, s2 = yf.sum((0, 2, 3)), (yf * yf).sum((0, 2, 3))
    assert (stats[0] - s1).abs().max().item() <= 1e-3 * s1.abs().max().item() + 0.05
    assert (stats[1] - s2).abs().max().item() <= 1e-3 * s2.abs().max().item() + 0.05
    # without statistics
    y2 = C.conv_fprop(x, w, stride, pad)
    assert torch.equal(y, y2)


@pytest.mark.parametrize("N,Ci,Co,HW,k", [(8, 16, 16, 32, 3), (4, 32, 32, 16, 3), (5, 64, 64, 8, 3), (4, 16, 32, 32, 1), (2, 32, 16, 16, 3),
                                          (2, 16, 64, 64, 3), (3, 32, 16, 28, 3), (2, 64, 32, 7, 3), (12, 64, 64, 64, 3)])
def test_conv_dgrad_tensor_core(C, N, Ci, Co, HW, k):
    torch.manual_seed(13)
    pad = k // 2
    assert C.conv_dgrad_supported(N, HW, HW, Ci, Co, k, 1, pad)
    dy = torch.randn(N, Co, HW, HW, device="cuda").bfloat16().contiguous(memory_format=torch.channels_last)
    w = (torch.randn(Co, Ci, k, k, device="cuda") * 0.1).bfloat16().contiguous(memory_format=torch.channels_last)
    dx = C.conv_dgrad(dy, w, 1, pad)
    torch.cuda.synchronize()
    assert C.read_status(0) == 0
    ref = torch.nn.grad.conv2d_input((N, Ci, HW, HW), w.float(), dy.float(), stride=1, padding=pad)
    assert dx.shape == ref.shape and dx.is_contiguous(memory_format=torch.channels_last)
    err = (dx.float() - ref).abs().max().item()
    assert err <= 0.01 * ref.abs().max().item() + 0.01, f"max err {err} (ref max {ref.abs().max().item()})"


def test_conv_fprop_dgrad_reject_unsupported(C):
    assert not C.conv_fprop_supported(4, 32, 32, 3, 16, 3, 1, 1)       # 3-channel stem
    assert not C.conv_fprop_supported(4, 28, 28, 16, 32, 3, 2, 1)      # strided, width not a power of two
    assert not C.conv_fprop_supported(4, 4, 4, 32, 64, 3, 2, 1)        # strided, fewer than 64 output pixels per image
    assert not C.conv_fprop_supported(4, 32, 32, 16, 16, 5, 1, 2)      # 5x5
    assert not C.conv_dgrad_supported(4, 32, 32, 16, 32, 3, 2, 1)      # strided data gradient



def test_bn_from_conv_sums_matches_stats_pass(C):
    torch.manual_seed(14)
    N, Ci, Co, HW = 16, 16, 32, 32
    x = torch.randn(N, Ci, HW, HW, device="cuda").bfloat16().contiguous(memory_format=torch.channels_last)
    w = (torch.randn(Co, Ci, 3, 3, device="cuda") * 0.1).bfloat16().contiguous(memory_format=torch.channels_last)
    res = torch.randn(N, Co, HW, HW, device="cuda").bfloat16().contiguous(memory_format=torch.channels_last)
    gamma, beta = torch.rand(Co, device="cuda") + 0.5, torch.randn(Co, device="cuda")
    sums = torch.zeros(2, Co, device="cuda")
    y = C.conv_fprop(x, w, 1, 1, sums)
    rm1, rv1 = torch.zeros(Co, device="cuda"), torch.ones(Co, device="cuda")
    rm2, rv2 = rm1.clone(), rv1.clone()
    o1, m1, r1 = C.bn_fwd(y, res, gamma, beta, rm1, rv1, 1e-5, 0.1, True, True)
    o2, m2, r2 = C.bn_fwd(y, res, gamma, beta, rm2, rv2, 1e-5, 0.1, True, True, sums)
    torch.cuda.synchronize()
    assert (m1 - m2).abs().max().item() < 1e-4
    assert ((r1 - r2).abs() / r1.abs()).max().item() < 1e-3
    assert (rm1 - rm2).abs().max().item() < 1e-4 and (rv1 - rv2).abs().max().item() < 1e-3
    assert (o1.float() - o2.float()).abs().max().item() <= 0.04


def test_eager_adam_on_unflattened_parameters_matches_torch(C):
    from flodl_b200 import nn
    torch.manual_seed(15)
    shapes = [(33, 17), (64,), (5, 4, 3)]
    ours = [nn.Parameter(torch.randn(*s, device="cuda"), f"p{i}") for i, s in enumerate(shapes)]
    ref = [p.t.detach().clone().requires_grad_(True) for p in ours]
    opt, ropt = nn.Adam(ours, 0.01), torch.optim.Adam(ref, lr=0.01)
    for step in range(3):
        for p, r in zip(ours, ref):
            g = torch.randn_like(r)
            p.t.grad = g.clone()
            r.grad = g.clone()
        opt.step()
        ropt.step()
    for p, r in zip(ours, ref):
        assert (p.t.detach() - r.detach()).abs().max().item() < 1e-5


@pytest.mark.parametrize("config", [0, 2])
def test_gemm_device_side_row_and_reduction_counts(C, config):
    """`m_dyn` / `k_dyn`: the kernel works on the device-side counts, buffers keep their static size."""
    torch.manual_seed(11)
    M, N, K, m_act = 1024, 512, 256, 300
    a = torch.randn(M, K, device="cuda").bfloat16()
    b = torch.randn(N, K, device="cuda").bfloat16()
    out = torch.full((M, N), 7.0, device="cuda", dtype=torch.bfloat16)
    cnt = torch.tensor([m_act], device="cuda", dtype=torch.int32)
    C.clear_status(0)
    C.gemm(a, b, out, False, False, config=config, m_dyn=cnt)
    torch.cuda.synchronize()
    assert C.read_status(0) == 0
    ref = a.float() @ b.float().t()
    assert (out[:m_act].float() - ref[:m_act]).abs().max().item() <= 0.02 * ref.abs().max().item() + 0.05
    tile_m = 256 if config == 0 else 128
    first_untouched = (m_act + tile_m - 1) // tile_m * tile_m
    assert torch.all(out[first_untouched:] == 7.0), "tiles past the dynamic row count must not be written"
    # reduction length: dW[n, k] = sum_t dy[t, n] x[t, k] over the first k_act rows only (rows up to the
    # next multiple of 64 are zero, as the producers of such operands guarantee)
    T, k_act = 1024, 200
    dy = torch.randn(T, 384, device="cuda").bfloat16()
    x = torch.randn(T, 256, device="cuda").bfloat16()
    dy[k_act:256] = 0
    x[k_act:256] = 0
    dw = torch.zeros(384, 256, device="cuda")
    kc = torch.tensor([k_act], device="cuda", dtype=torch.int32)
    C.gemm(dy, x, dw, True, True, config=config, accumulate=True, k_dyn=kc)
    torch.cuda.synchronize()
    assert C.read_status(0) == 0
    ref = dy[:k_act].float().t() @ x[:k_act].float()
    assert (dw - ref).abs().max().item() <= 0.02 * ref.abs().max().item() + 0.05
    # a zero count leaves the output alone
    dw2 = torch.full((384, 256), 3.0, device="cuda")
    C.gemm(dy, x, dw2, True, True, config=config, accumulate=True, k_dyn=torch.zeros(1, device="cuda", dtype=torch.int32))
    torch.cuda.synchronize()
    assert torch.all(dw2 == 3.0)


def test_row_compaction_kernels(C):
    torch.manual_seed(5)
    rows, cols = 3000, 136
    tgt = torch.randint(0, 50, (rows,), device="cuda")
    tgt[torch.rand(rows, device="cuda") < 0.8] = -100
    idx, tc, counts = C.compact_targets(tgt, -100)
    n, n_pad = counts.tolist()
    act = (tgt != -100).nonzero().flatten()
    assert n == act.numel() and n_pad == min(rows, (n + 255) // 256 * 256)
    assert torch.equal(idx[:n].long(), act) and torch.equal(tc[:n], tgt[act]) and torch.all(tc[n:] == -100)
    x = torch.randn(rows, cols, device="cuda").bfloat16()
    xc = torch.full_like(x, 9.0)
    C.gather_rows(x, idx, counts, xc)
    assert torch.equal(xc[:n], x[act]) and torch.all(xc[n:n_pad] == 0) and torch.all(xc[n_pad:] == 9.0)
    dx = torch.zeros_like(x)
    C.scatter_rows(xc, idx, counts, dx)
    ref = torch.zeros_like(x)
    ref[act] = x[act]
    assert torch.equal(dx, ref)
    # nothing active
    idx, tc, counts = C.compact_targets(torch.full((700,), -100, device="cuda"), -100)
    assert counts.tolist() == [0, 0]


def test_masked_lm_loss_on_labelled_rows_only_matches_full_projection():
    """The masked-LM head projects only the labelled rows; loss and every gradient must agree with the
    projection of all rows (ignored rows contribute nothing to either)."""
    from flodl_b200 import ops
    torch.manual_seed(9)
    rows, K, V = 2048, 256, 3000
    x0 = (torch.randn(rows, K, device="cuda") * 0.5).bfloat16()
    w0 = (torch.randn(V, K, device="cuda") * 0.05)
    b0 = torch.randn(V, device="cuda") * 0.1
    tgt = torch.randint(0, V, (rows,), device="cuda")
    tgt[torch.rand(rows, device="cuda") < 0.85] = -100
    res = []
    for sparse in (False, True):
        x, w, b = x0.clone().requires_grad_(True), w0.clone().requires_grad_(True), b0.clone().requires_grad_(True)
        loss = ops.linear_cross_entropy(x, w, b, tgt, -100, sparse_targets=sparse)
        (loss * 1.5).backward()
        torch.cuda.synchronize()
        res.append((loss.item(), x.grad.float(), w.grad.float(), b.grad.float()))
    (l0, dx0, dw0, db0), (l1, dx1, dw1, db1) = res
    assert abs(l0 - l1) < 1e-4 * max(1.0, abs(l0)), (l0, l1)
    assert torch.equal(dx1[tgt == -100], torch.zeros_like(dx1[tgt == -100]))
    for a, b_, name in ((dx0, dx1, "dx"), (dw0, dw1, "dw"), (db0, db1, "db")):
        scale = a.abs().max().item() + 1e-12
        assert (a - b_).abs().max().item() <= 2e-2 * scale, (name, (a - b_).abs().max().item(), scale)
    # against fp32 PyTorch
    xr, wr, br = x0.float().requires_grad_(True), w0.clone().requires_grad_(True), b0.clone().requires_grad_(True)
    ref = F.cross_entropy(F.linear(xr, wr.bfloat16().float(), br), tgt, ignore_index=-100)
    (ref * 1.5).backward()
    assert abs(ref.item() - l1) < 5e-2      # bf16 logits against an fp32 projection
    assert (wr.grad - dw1).abs().max().item() <= 3e-2 * wr.grad.abs().max().item() + 1e-4


def test_bounds_checked_debug_build_records_instead_of_faulting():
    """The debug library (`FLODL_B200_BOUNDS_CHECK=1`, built beside the regular one) range-checks every
    index a kernel reads from device memory; see tests/_bounds_worker.py for the sweep."""
    import os
    import subprocess
    import sys
    here = os.path.dirname(os.path.abspath(__file__))
    env = dict(os.environ, FLODL_B200_BOUNDS_CHECK="1")
    res = subprocess.run([sys.executable, os.path.join(here, "_bounds_worker.py")], capture_output=True, text=True, timeout=900, env=env)
    assert res.returncode == 0 and "BOUNDS_OK" in res.stdout, res.stdout[-2000:] + res.stderr[-3000:]


@pytest.mark.parametrize("rows,N,K,bias,dtype,order", [(77, 128, 256, "bf16", "bf16", "rows"), (1, 64, 64, None, "bf16", "rows"), (1500, 192, 128, "fp32", "fp32", "rows"),
                                                      (200, 72, 40, "bf16", "bf16", "columns"), (130, 128, 64, "fp32", "bf16", "strided")])
def test_packed_linear_without_gradients(C, rows, N, K, bias, dtype, order):
    """The grouped projections against the general path (one `linear` each under autograd, stacked), over sizes that take one launch and sizes
    that take three, input orders, and types. The same products in another order of summation: one rounding to bf16 apart."""
    from flodl_b200 import nn, ops
    from flodl_b200.ops import core
    torch.manual_seed(16)
    dt = torch.bfloat16 if dtype == "bf16" else torch.float32
    x = torch.randn(rows, K, device="cuda").to(dt)
    if order == "columns":
        x = x.t().contiguous().t()
    elif order == "strided":
        x = torch.cat((x, x), 1)[:, K:]
    ws = [(torch.randn(N, K, device="cuda") / math.sqrt(K)).to(dt).requires_grad_() for _ in range(3)]
    bt = {"bf16": torch.bfloat16, "fp32": torch.float32}.get(bias)
    bs = [None if bias is None else torch.randn(N, device="cuda").to(bt).requires_grad_() for _ in range(3)]
    was = core.eager_min_numel()
    core.set_eager_min_numel(0)
    try:
        with nn.AutocastGuard(torch.bfloat16):
            want = ops.packed_linear(x, ws, bs)
            with torch.no_grad():
                got = ops.packed_linear(x, ws, bs)
                ffn = ops.feed_forward(x, ws[0], bs[0], torch.eye(N, device="cuda").to(dt), None)
                norm = ops.layer_norm(got[:, 0], torch.ones(N, device="cuda").to(dt), torch.zeros(N, device="cuda").to(dt), residual=got[:, 1])
            ref = ops.layer_norm(want[:, 0], torch.ones(N, device="cuda"), torch.zeros(N, device="cuda"), residual=want[:, 1])
    finally:
        core.set_eager_min_numel(was)
    assert want.requires_grad and not got.requires_grad and got.shape == want.shape == (rows, 3, N) and got.dtype == want.dtype
    close = lambda a, b, u: ((a.double() - b.double()).norm() / b.double().norm()).item() < u
    assert close(got, want, 2 ** -8) and close(norm, ref, 2 ** -7)
    act = torch.nn.functional.gelu(want[:, 0].detach().double())
    assert close(ffn, act, 2 ** -7)


def test_first_calls_of_a_process_under_capture():
    """An eager step of small tensors runs no native kernel, so that a process may meet its first one while it captures: the calls that set a thread
    or a device up have to be legal there, and the status word must not be part of the graph."""
    code = """
import torch
from flodl_b200 import _ext
C = _ext.require()
a, b = torch.randn(200, 128, device="cuda").bfloat16(), torch.randn(64, 128, device="cuda").bfloat16()
q, k, v = torch.randn(1, 300, 3, 2, 64, device="cuda").bfloat16().unbind(2)
out = torch.zeros(200, 64, device="cuda", dtype=torch.bfloat16)
torch.cuda.synchronize()
g = torch.cuda.CUDAGraph()
with torch.cuda.graph(g, capture_error_mode="thread_local"):
    C.gemm(a, b, out)
    o, lse = C.attn_fwd(q, k, v, None, 0.125, False)
assert C.read_status(0) == 0
g.replay()
torch.cuda.synchronize()
assert C.read_status(0) == 0
ref = a.double() @ b.double().t()
assert ((out.double() - ref).norm() / ref.norm()).item() < 2 ** -8
s = torch.softmax(torch.einsum("bqhd,bkhd->bhqk", q.double(), k.double()) * 0.125, -1)
ref = torch.einsum("bhqk,bkhd->bqhd", s, v.double())
assert ((o.double() - ref).norm() / ref.norm()).item() < 2 ** -8
print("CAPTURE_OK")
"""
    import os
    import subprocess
    import sys
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    res = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300, cwd=root)
    assert res.returncode == 0 and "CAPTURE_OK" in res.stdout, res.stdout[-2000:] + res.stderr[-3000:]
