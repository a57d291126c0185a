"""tcgen05 GEMM against an fp32 PyTorch reference (and its fused epilogues)."""
import ctypes

import pytest
import torch

from pie_b200 import ops
from pie_b200.ops import _lib, reference as ref

pytestmark = pytest.mark.gpu
DEV = "cuda"


def bf(*shape, scale=1.0, seed=0):
    g = torch.Generator(device=DEV).manual_seed(seed)
    return (torch.randn(*shape, generator=g, device=DEV) * scale).to(torch.bfloat16)


def check(y, want, k):
    err = (y.float() - want.float()).abs().max().item()
    # bf16 output rounding (2^-8 relative) + fp32 accumulation over k terms
    tol = 2e-2 * want.float().abs().max().item() + 1e-3 * k ** 0.5
    assert err <= tol, f"max err {err} > {tol}"
    ops.check_kernel_status()


@pytest.mark.parametrize("m,n,k", [(128, 256, 64), (128, 256, 512), (256, 512, 4096), (1, 6144, 4096),
                                   (77, 4096, 4096), (512, 6144, 4096), (300, 1000, 328), (2048, 14336, 4096),
                                   (130, 128256, 256)])
@pytest.mark.parametrize("bn", [0, 64, 128, 256])
def test_gemm_plain(m, n, k, bn):
    if bn and (m * n > 4096 * 4096) and bn != 256:
        pytest.skip("large shape only with the automatic tile choice")
    x, w = bf(m, k, seed=1), bf(n, k, scale=0.05, seed=2)
    y = ops.gemm(x, w, force_bn=bn)
    check(y, x.float() @ w.float().t(), k)


@pytest.mark.parametrize("m,n,k", [(512, 6144, 4096), (512, 4096, 14336), (512, 768, 4096), (64, 4096, 4096),
                                   (300, 2048, 8192), (512, 28672, 4096)])
@pytest.mark.parametrize("epi", ["store", "residual", "swiglu"])
def test_gemm_stream_k_matches_whole_tile_and_reference(m, n, k, epi):
    """Skinny shapes take the stream-K schedule (split tiles fixed up through the workspace);
    force_bn=-1 forces whole-tile scheduling of the same kernel."""
    x, w = bf(m, k, seed=11), bf(n, k, scale=0.03, seed=12)
    r = bf(m, n, seed=13) if epi == "residual" else None
    e = {"store": ops.EPI_STORE, "residual": ops.EPI_RESIDUAL, "swiglu": ops.EPI_SWIGLU}[epi]
    for rep in range(2):     # twice: the arrival counters must be back at zero
        y = ops.gemm(x, w, residual=r, epilogue=e)
    y_dp = ops.gemm(x, w, residual=r, epilogue=e, force_bn=-1)
    want = x.float() @ w.float().t()
    if epi == "residual":
        want = want + r.float()
    if epi == "swiglu":
        want = ref.swiglu_interleaved(want)
    check(y, want, k)
    check(y_dp, want, k)


def route(m, n, k):
    """(CTA pairs or single CTAs, tile width, pairs or CTAs, K split) of a product of more than 128 rows."""
    out = (ctypes.c_int * 4)()
    assert _lib.declare("pie_gemm_route", [ctypes.c_int] * 5 + [ctypes.c_void_p])(m, n, k, ops.num_sms(DEV), 1, out) == 0
    return tuple(out)


@pytest.mark.parametrize("m,n,k,taken", [(200, 1024, 4096, True), (512, 768, 4096, True), (300, 2048, 8192, True), (1024, 512, 4096, True),
                                         (257, 1536, 4104, True), (512, 4096, 14336, False), (64, 4096, 4096, False)])
@pytest.mark.parametrize("epi", ["store", "residual", "swiglu"])
def test_gemm_single_ctas_split_k(m, n, k, taken, epi):
    """K split evenly over single CTAs, several row tiles or one, parts of two and more CTAs per tile, ragged ends: against the fp32
    reference and whole tiles of the same kernel. `taken`: the products that run like this by themselves. 32-bit sums of one product
    differ by their order alone: one rounding to bf16 (2^-9), or two with a GLU's own error, of values near 1."""
    plan = (ctypes.c_int * 3)()
    assert _lib.declare("pie_gemm_plan", [ctypes.c_int] * 5 + [ctypes.c_void_p])(m, n, k, ops.num_sms(DEV), 1, plan) == 0
    assert plan[2] == 1
    assert not taken or route(m, n, k) == (0, *plan)
    x, w = bf(m, k, seed=71), bf(n, k, scale=k ** -0.5, seed=72)
    r = bf(m, n, seed=73) if epi == "residual" else None
    e = {"store": ops.EPI_STORE, "residual": ops.EPI_RESIDUAL, "swiglu": ops.EPI_SWIGLU}[epi]
    default = ops.gemm(x, w, residual=r, epilogue=e)
    ops.set_gemm_pairs(False)
    ops.set_gemm_swap(0)
    try:
        got = [ops.gemm(x, w, residual=r, epilogue=e) for _ in range(3)]        # again: the arrival counters must be back at zero
        whole = ops.gemm(x, w, residual=r, epilogue=e, force_bn=-1)
    finally:
        ops.set_gemm_pairs(True)
        ops.set_gemm_swap(128)
    ops.check_kernel_status()
    assert torch.equal(got[0], got[1]) and torch.equal(got[0], got[2])
    assert not taken or torch.equal(got[0], default)
    want = x.float() @ w.float().t()
    if epi == "residual":
        want = want + r.float()
    if epi == "swiglu":
        want = ref.swiglu_interleaved(want)
    for y in (got[0], whole):
        torch.testing.assert_close(y.float(), want, rtol=2 ** -8, atol=2e-3)


@pytest.mark.parametrize("m,n,k,pairs", [(640, 65536, 256, 0), (1024, 49152, 256, 0), (640, 7168, 128, 0), (385, 18944, 128, 0),
                                         (2305, 28672, 256, 0),
                                         (512, 9216, 512, 0), (640, 7168, 2048, 0), (300, 12288, 4096, 0), (257, 12288, 2048, 0),
                                         (129, 24576, 4096, 1), (200, 20480, 4096, 1), (129, 24576, 5120, 1), (300, 4096, 4096, 1),
                                         (300, 16384, 4096, 1),
                                         (512, 512, 1024, 1), (512, 4096, 4096, 1), (2305, 28672, 4096, 1), (200, 49152, 2048, 1)])
def test_gemm_products_run_on_the_kernel_that_takes_less_time(m, n, k, pairs):
    """Shapes at which one of the two kernels for more than 128 rows was measured 8 to 40 % faster on 148 SMs; either gives the same bits."""
    out = (ctypes.c_int * 4)()
    assert _lib.declare("pie_gemm_route", [ctypes.c_int] * 5 + [ctypes.c_void_p])(m, n, k, 148, 1, out) == 0
    assert out[0] == pairs and out[3] == 0
    if m * n < 1 << 25:
        x, w = bf(m, k, seed=58), bf(n, k, scale=k ** -0.5, seed=59)
        width = _lib.declare("pie_gemm_set_pair_width", [ctypes.c_int])
        width(-1)
        try:
            y = ops.gemm(x, w)
        finally:
            width(0)
        assert torch.equal(y, ops.gemm(x, w, force_bn=-1)) and torch.equal(y, ops.gemm(x, w))
        ops.check_kernel_status()


def product32(x, w, out=None, width=0):
    """out (0 if not given) + x @ w.T in 32 bits; `width`: in whole tiles of that width on CTA pairs."""
    out = torch.zeros(x.shape[0], w.shape[0], device=DEV) if out is None else out
    fn = _lib.declare("pie_gemm_bf16_stream", [ctypes.c_void_p] * 5 + [ctypes.c_int, ctypes.c_void_p] + [ctypes.c_int] * 6 +
                      [ctypes.c_void_p, ctypes.c_int, ctypes.c_void_p])
    set_width = _lib.declare("pie_gemm_set_pair_width", [ctypes.c_int])
    ops.ensure_gemm_workspace(DEV)
    set_width(width)
    try:
        assert fn(x.data_ptr(), w.data_ptr(), None, out.data_ptr(), out.data_ptr(), out.stride(0), None, x.shape[0], w.shape[0], x.shape[1],
                  x.stride(0), w.stride(0), 0, ops.kernel_status(DEV).data_ptr(), ops.num_sms(DEV),
                  torch.cuda.current_stream().cuda_stream) == 0
    finally:
        set_width(0)
    return out


@pytest.mark.parametrize("m,n,k", [(512, 4096, 14336), (256, 5120, 8192), (1030, 6144, 4096), (200, 28672, 4096), (385, 10240, 5120)])
def test_gemm_pairs_add_up_the_parts_of_a_split_k_in_order(m, n, k):
    """Large products whose last round of tiles would be short: K split evenly over the pairs. Bit for bit the sum of the parts, each a
    chain of its own, in their order - the order these products have always had."""
    assert route(m, n, k) == (1, 256, 74, 1)
    x, w = bf(m, k, seed=61), bf(n, k, scale=k ** -0.5, seed=62)
    got = [product32(x, w) for _ in range(2)]              # twice: the arrival counters must be back at zero
    assert torch.equal(*got)
    tiles_m, tiles_n, blocks = -(-m // 256), -(-n // 256), -(-k // 64)
    total = tiles_m * tiles_n * blocks
    starts = [total * p // 74 for p in range(75)]
    for tile in {0, tiles_m * tiles_n // 2, tiles_m * tiles_n - 1}:
        r, c = tile % tiles_m * 256, tile // tiles_m * 256
        cuts = sorted({tile * blocks, (tile + 1) * blocks, *(s for s in starts if tile * blocks < s < (tile + 1) * blocks)})
        want = None
        for a, b in zip(cuts, cuts[1:]):
            a, b = (a - tile * blocks) * 64, min(k, (b - tile * blocks) * 64)
            want = product32(x[:, a:b], w[c:c + 256, a:b], want, width=256)
        assert torch.equal(got[0][r:r + 256, c:c + 256], want[r:r + 256]), tile
    ops.check_kernel_status()


@pytest.mark.parametrize("m,n,k", [(512, 4096, 14336), (256, 7168, 8192), (129, 4096, 14336), (300, 1024, 8192), (1024, 3072, 8192),
                                   (640, 512, 4096)])
def test_gemm_split_k_keeps_the_error_of_its_shorter_chains(m, n, k):
    """Additions of the tensor cores are cut off, so a sum's error grows with its chain. Products whose K is split, on pairs or on single
    CTAs, have chains of less than half of K and keep 0.6 of the whole chain's error or less; 300 x 1024 x 8192 has 0.14."""
    assert route(m, n, k)[3] == 1
    x, w = bf(m, k, seed=63), bf(n, k, scale=k ** -0.5, seed=64)
    want = x.double() @ w.double().t()
    err = [float((y.double() - want).norm()) for y in (product32(x, w), product32(x, w, width=128))]
    assert err[0] <= 0.6 * err[1]
    ops.check_kernel_status()


def test_gemm_residual():
    m, n, k = 333, 4096, 1024
    x, w, r = bf(m, k, seed=3), bf(n, k, scale=0.05, seed=4), bf(m, n, seed=5)
    y = ops.gemm(x, w, residual=r, epilogue=ops.EPI_RESIDUAL)
    check(y, x.float() @ w.float().t() + r.float(), k)


def test_gemm_swiglu():
    m, n, k = 200, 2 * 1408, 512
    x, w = bf(m, k, seed=6), bf(n, k, scale=0.05, seed=7)
    y = ops.gemm(x, w, epilogue=ops.EPI_SWIGLU)
    want = ref.swiglu_interleaved((x.float() @ w.float().t()))
    assert y.shape == (m, n // 2)
    check(y, want, k)


def test_gemm_strided_operands():
    m, n, k = 96, 512, 256
    big = bf(m, 3 * k, seed=8)
    x = big[:, k:2 * k]                      # row stride 3k
    w = bf(n, k, scale=0.05, seed=9)
    out = torch.zeros(m, 2 * n, dtype=torch.bfloat16, device=DEV)
    ops.gemm(x, w, out=out[:, n:])
    check(out[:, n:], x.float() @ w.float().t(), k)
    assert float(out[:, :n].abs().max()) == 0.0


@pytest.mark.parametrize("bn", [16, 48, 80, 112, 176, 208, 240])
@pytest.mark.parametrize("epi", ["store", "residual", "swiglu"])
def test_gemm_odd_tile_widths(bn, epi):
    """Tile widths between the native 64/128/256 (chosen to fill the machine's waves): the last
    tile of a row is ragged and the SwiGLU epilogue halves the column index."""
    m, n, k = 200, 2000 if epi != "swiglu" else 2016, 1024
    x, w = bf(m, k, seed=21), bf(n, k, scale=0.04, seed=22)
    r = bf(m, n, seed=23) if epi == "residual" else None
    e = {"store": ops.EPI_STORE, "residual": ops.EPI_RESIDUAL, "swiglu": ops.EPI_SWIGLU}[epi]
    ops.set_gemm_pairs(False)
    try:
        y = ops.gemm(x, w, residual=r, epilogue=e, force_bn=-bn)
    finally:
        ops.set_gemm_pairs(True)
    want = x.float() @ w.float().t()
    if epi == "residual":
        want = want + r.float()
    if epi == "swiglu":
        want = ref.swiglu_interleaved(want)
    check(y, want, k)


@pytest.mark.parametrize("bn", [64, 80, 96, 112, 144, 160, 176, 208, 224, 256])
@pytest.mark.parametrize("m,n,k", [(129, 128, 64), (256, 1000, 72), (257, 1032, 520), (700, 2080, 1096), (2305, 520, 136), (1025, 9216, 256)])
@pytest.mark.parametrize("epi", ["store", "residual", "swiglu"])
def test_gemm_pair_tile_widths(bn, m, n, k, epi):
    """CTA-pair tiles of every kind of width (last chunk of the epilogue whole or not, fewer columns than a chunk), one or more tiles
    per pair, ragged ends of all three sizes. 32-bit sums of one product differ by their order alone: one rounding to bf16 (2^-9), or
    two with a GLU's own error, of values near 1."""
    if epi == "swiglu":
        n = n // 32 * 32
    x, w = bf(m, k, seed=51), bf(n, k, scale=k ** -0.5, seed=52)
    r = bf(m, n, seed=53) if epi == "residual" else None
    e = {"store": ops.EPI_STORE, "residual": ops.EPI_RESIDUAL, "swiglu": ops.EPI_SWIGLU}[epi]
    width = _lib.declare("pie_gemm_set_pair_width", [ctypes.c_int])
    width(bn)
    try:
        y = ops.gemm(x, w, residual=r, epilogue=e)
    finally:
        width(0)
    want = x.float() @ w.float().t()
    if epi == "residual":
        want = want + r.float()
    if epi == "swiglu":
        want = ref.swiglu_interleaved(want)
    ops.check_kernel_status()
    torch.testing.assert_close(y.float(), want, rtol=2 ** -8, atol=2e-3)


@pytest.mark.parametrize("bn", [64, 80, 112, 144, 176, 208, 256])
@pytest.mark.parametrize("m,n,k", [(129, 128, 64), (257, 1056, 520), (700, 2080, 1096), (2305, 544, 136)])
@pytest.mark.parametrize("epi", ["geglu", "xielu", "stream"])
def test_gemm_pair_tile_widths_of_the_other_epilogues(bn, m, n, k, epi):
    """As above for the epilogues with an activation or a bias and for the 32-bit stream, whose 128-byte pieces end inside a chunk. Sums of
    1096 or fewer in 32 bits: 69 additions cut off at 2^-23 of partial sums below 4 are 3.3e-5; bf16 results are one rounding (2^-9), or
    two with an activation's own error, of values near 1."""
    from pie_b200.ops import latent as lops
    x, w, b = bf(m, k, seed=54), bf(n, k, scale=k ** -0.5, seed=55), bf(n, seed=56)
    act = torch.tensor([0.3, -0.2], dtype=torch.bfloat16, device=DEV)
    stream = torch.randn(m, n, device=DEV, generator=torch.Generator(device=DEV).manual_seed(57))
    z = x.double() @ w.double().t()
    width = _lib.declare("pie_gemm_set_pair_width", [ctypes.c_int])
    width(bn)
    try:
        if epi == "geglu":
            y, want = ops.gemm(x, w, epilogue=ops.EPI_GEGLU), ref.glu_interleaved(z.float(), "gelu_tanh").double()
        elif epi == "xielu":
            y = lops.gemm_xielu(x, w, b, act, torch.full((m, n), 7.0, dtype=torch.bfloat16, device=DEV))
            z = z + b.double()
            pos, neg = torch.nn.functional.softplus(act.double())
            want = torch.where(z > 0, pos * z * z, (0.5 + neg) * (torch.expm1(z) - z)) + 0.5 * z
        else:
            y, copy = lops.gemm_stream(x, w, b, stream.clone(), copy=True)
            want = stream.double() + z + b.double()
    finally:
        width(0)
    ops.check_kernel_status()
    if epi == "stream":
        torch.testing.assert_close(y.double(), want, rtol=2 ** -22, atol=3.3e-5)
        assert torch.equal(copy, y.to(torch.bfloat16))
    else:
        torch.testing.assert_close(y.double(), want, rtol=2 ** -8, atol=2e-3)


def tp_args(world, rank, rows, n, epoch):
    """Arguments of a tensor-parallel product on one GPU: every rank's receive buffer and flags are buffers of this GPU, and the flags that
    the gate looks at are already raised."""
    t = dict(recv=torch.full((world, world, rows, n), 7.0, dtype=torch.bfloat16, device=DEV),
             rs_flags=torch.zeros(world, 8, dtype=torch.int32, device=DEV), ag_flags=torch.full((8,), epoch, dtype=torch.int32, device=DEV),
             counters=torch.tensor([0, 0, 0, epoch], dtype=torch.int32, device=DEV))       # rs_done, rs_epoch, -, ag_epoch
    blob = ctypes.create_string_buffer(_lib.declare("pie_tp_args_size", [])())
    fill = _lib.declare("pie_tp_fill_args", [ctypes.c_void_p] * 7 + [ctypes.c_int] * 4)
    each = lambda x: (ctypes.c_void_p * world)(*[x[i].data_ptr() for i in range(world)])
    c = t["counters"].data_ptr()
    assert fill(blob, t["ag_flags"].data_ptr(), c + 12, each(t["recv"]), each(t["rs_flags"]), c, c + 4, world, rank, rows, 0) == 0
    return blob, t


def gemm_tp(x, w, out, epilogue, blob, rows, gated):
    fn = _lib.declare("pie_gemm_bf16_tp", [ctypes.c_void_p] * 3 + [ctypes.c_int] * 7 + [ctypes.c_void_p] + [ctypes.c_int] * 3 +
                      [ctypes.c_void_p, ctypes.c_int, ctypes.c_void_p])
    ops.ensure_gemm_workspace(DEV)
    assert fn(x.data_ptr(), w.data_ptr(), None if out is None else out.data_ptr(), x.shape[0], w.shape[0], x.shape[1], x.stride(0), w.stride(0),
              0 if out is None else out.stride(0), epilogue, blob, rows, gated, 0, ops.kernel_status(DEV).data_ptr(), ops.num_sms(DEV),
              torch.cuda.current_stream().cuda_stream) == 0


@pytest.mark.parametrize("bn,m,n,k", [(64, 129, 128, 64), (80, 700, 1032, 520), (112, 1025, 2080, 264), (176, 385, 4096, 1096),
                                      (208, 2305, 520, 136), (256, 300, 1000, 512), (0, 512, 4096, 14336), (0, 200, 28672, 4096),
                                      (0, 512, 4096, 4096), (0, 200, 1024, 4096)])
@pytest.mark.parametrize("world", [1, 3])
def test_gemm_pairs_scatter_rows_to_owners_and_wait_at_the_gate(bn, m, n, k, world):
    """The tensor-parallel forms on pairs, whole tiles of many widths and K split (width 0: as planned), right behind the product that
    writes their activations: the rows of every owner are those of the plain product bit for bit, in their place and nowhere else, the
    last arrival resets its counter and raises the flags; a gate whose flags are up lets the plain product through."""
    rank, rows = world - 1, -(-m // world // 32) * 32 + 32
    first, square, w = bf(m, 256, seed=74), bf(k, 256, scale=1 / 16, seed=75), bf(n, k, scale=k ** -0.5, seed=76)
    blob, t = tp_args(world, rank, rows, n, 5)
    width = _lib.declare("pie_gemm_set_pair_width", [ctypes.c_int])
    width(bn)
    try:
        want = ops.gemm(ops.gemm(first, square), w)
        torch.cuda.synchronize()
        for turn in range(2):
            gemm_tp(ops.gemm(first, square), w, None, 3, blob, rows, 0)
        gated = [torch.empty_like(want) for _ in range(2)]
        for out, owned in zip(gated, (rows, 0)):
            gemm_tp(ops.gemm(first, square), w, out, ops.EPI_STORE, blob, owned, 1)
    finally:
        width(0)
    torch.cuda.synchronize()
    ops.check_kernel_status()
    assert torch.equal(gated[0], want) and torch.equal(gated[1], want)
    expect = torch.full_like(t["recv"], 7.0)
    for o in range(world):
        mine = want[o * rows:(o + 1) * rows]
        expect[o, rank, :len(mine)] = mine
    assert torch.equal(t["recv"], expect)
    assert t["counters"].tolist() == [0, 2, 0, 5] and t["rs_flags"][:, rank].tolist() == [2] * world


@pytest.mark.parametrize("m", [1, 7, 64, 65, 100, 128])
@pytest.mark.parametrize("n,k", [(6144, 4096), (4096, 14336), (1000, 512), (28672, 4096)])
@pytest.mark.parametrize("epi", ["store", "residual", "swiglu"])
def test_gemm_swapped_operands_small_batch(m, n, k, epi):
    """Batches of at most 128 rows run C^T = W A^T (weights on the 128-row side, transposed epilogue):
    same result as the direct orientation and as the fp32 reference, ragged feature counts included."""
    if epi == "swiglu" and n % 32:
        n = 992
    x, w = bf(m, k, seed=31), bf(n, k, scale=0.03, seed=32)
    r = bf(m, n, seed=33) if epi == "residual" else None
    e = {"store": ops.EPI_STORE, "residual": ops.EPI_RESIDUAL, "swiglu": ops.EPI_SWIGLU}[epi]
    ops.set_gemm_swap(1000)      # every shape, not only those the selection rule picks
    try:
        y = ops.gemm(x, w, residual=r, epilogue=e)
        ops.set_gemm_swap(0)
        y0 = ops.gemm(x, w, residual=r, epilogue=e)
    finally:
        ops.set_gemm_swap(128)
    ref = x.float() @ w.float().t()
    if epi == "residual":
        ref = ref + r.float()
    if epi == "swiglu":
        ref = torch.nn.functional.silu(ref[:, 0::2]) * ref[:, 1::2]
    check(y, ref, k)
    check(y0, ref, k)
    ops.check_kernel_status()


@pytest.mark.parametrize("m", [1, 3, 17, 127, 129, 130, 200, 255, 257, 300])
@pytest.mark.parametrize("n,k,epi", [(1024, 4096, "store"), (28672, 512, "swiglu"), (1000, 520, "residual")])
def test_gemm_tiles_of_no_more_rows_than_the_batch_has(m, n, k, epi):
    """A tile's box ends with its rows; what shared memory holds beyond them (here infinities of the product before)
    reaches no stored row."""
    x, w = bf(m, k, seed=41), bf(n, k, scale=0.03, seed=42)
    r = bf(m, n, seed=43) if epi == "residual" else None
    e = {"store": ops.EPI_STORE, "residual": ops.EPI_RESIDUAL, "swiglu": ops.EPI_SWIGLU}[epi]
    want = x.float() @ w.float().t()
    if epi == "residual":
        want = want + r.float()
    if epi == "swiglu":
        want = ref.swiglu_interleaved(want)
    wild = torch.full((128, k), float("inf"), dtype=torch.bfloat16, device=DEV)
    for swap in (0, 128, 1000):
        ops.set_gemm_swap(swap)
        try:
            ops.gemm(wild, w)
            ops.set_gemm_pairs(swap != 0)
            y = ops.gemm(x, w, residual=r, epilogue=e)
        finally:
            ops.set_gemm_swap(128)
            ops.set_gemm_pairs(True)
        check(y, want, k)


@pytest.mark.parametrize("m,n,k", [(1, 4096, 2048), (100, 1024, 512), (40, 96, 256), (200, 256, 512), (300, 4096, 8192)])
def test_products_over_expanded_weights_of_one_shape(m, n, k):
    """Layers of one shape share the memory that their fp8 weights are expanded into: every product reads its own expansion."""
    x = bf(m, k, seed=51)
    layers = [ops.quantize_fp8_block(bf(n, k, scale=0.05, seed=52 + i).float()) for i in range(6)]
    want = [ops.gemm(x, q.dequant()) for q in layers]
    got = [ops.gemm_fp8w(x, q, mode="dequant") for _ in range(4) for q in layers]
    for i, y in enumerate(got):
        assert torch.equal(y, want[i % len(layers)])
    ops.check_kernel_status()


@pytest.mark.parametrize("n,k", [(256, 512), (1024, 1536), (1536, 1000), (4096, 768)])
def test_rows_are_the_same_in_the_kernel_for_small_batches(n, k):
    """Where K is not split (below 2048) a row's result is the same in a small batch's kernel and in the general one, in all epilogues:
    one order of sums, bias and residual included."""
    from pie_b200.ops import latent as lops
    x, w, r, b = bf(129, k, seed=61), bf(n, k, scale=0.03, seed=62), bf(129, n, seed=63), bf(n, seed=64)
    act = torch.tensor([0.3, -0.2], dtype=torch.bfloat16, device=DEV)
    stream = torch.randn(129, n, device=DEV, generator=torch.Generator(device=DEV).manual_seed(65)) * 3
    runs = {
        "store": lambda m: ops.gemm(x[:m], w),
        "residual": lambda m: ops.gemm(x[:m], w, residual=r[:m], epilogue=ops.EPI_RESIDUAL),
        "swiglu": lambda m: ops.gemm(x[:m], w, epilogue=ops.EPI_SWIGLU),
        "geglu": lambda m: ops.gemm(x[:m], w, epilogue=ops.EPI_GEGLU),
        "xielu": lambda m: lops.gemm_xielu(x[:m], w, b, act, torch.empty(m, n, dtype=torch.bfloat16, device=DEV)),
        "stream": lambda m: lops.gemm_stream(x[:m], w, b, stream[:m].clone())[0],
        "stream without bias": lambda m: lops.gemm_stream(x[:m], w, None, stream[:m].clone())[0],
    }
    for name, run in runs.items():
        if n % 32 and "glu" in name:
            continue
        large = run(129)
        for m, swap in ((1, 128), (40, 128), (128, 128), (128, 1000)):
            ops.set_gemm_swap(swap)
            try:
                small = run(m)
            finally:
                ops.set_gemm_swap(128)
            assert torch.equal(small, large[:m]), (name, m, int((small != large[:m]).sum()))
    ops.check_kernel_status()
