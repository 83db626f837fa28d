"""Parity of the CUDA kernels with the CPU oracle, through the C ABI (ctypes) and the Python
classes that mirror the reference.  Bars: dequantised tiles bit-exact; layer outputs
rel-L2 <= 1e-3 (fp16 storage, fp32 accumulation); the reference's own kernel-test bound
max|err| < 0.01 (inference/kernels/test_kernels.py:105) on its data distributions."""

import pytest
import torch

from oracle import glorcq_oracle as O
from tests import cases

pytestmark = pytest.mark.gpu
REL = 1e-3


@pytest.fixture(scope="module")
def dev():
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    from glorcq_b200 import _build
    _build.build()
    return torch.device("cuda:0")


# ---- tiles ---------------------------------------------------------------------------------
@pytest.mark.parametrize("N,K,bits,gs,int_zeros", [
    (1408, 2048, 2, 128, True), (2048, 1408, 2, 128, True), (40, 200, 2, 128, True), (17, 128, 2, 128, False),
    (64, 256, 4, 128, True), (2048, 2048, 4, 128, True), (33, 192, 4, 64, False), (48, 512, 2, 256, True)])
def test_gptq_tiles_bit_exact(dev, N, K, bits, gs, int_zeros):
    from glorcq_b200.tiled import TiledWeight
    d = cases.make_linear(101 + N + K, N, K, fmt="gptq", bits=bits, groupsize=gs, int_zeros=int_zeros, with_lora=False)
    tw = TiledWeight.from_gptq(d["qweight_int"].to(dev), d["scales"].to(dev), d["zeros"].to(dev), bits, gs)
    W = tw.dequantize().cpu()
    ref = O.gptq_tile_fp16(d["qweight_int"], d["scales"], d["zeros"], gs)
    assert torch.equal(W, ref)


@pytest.mark.parametrize("B", [1, 9, 32, 33])
@pytest.mark.parametrize("N,K,gs", [(2048, 2048, 128), (40, 192, 64)])
def test_3bit_codes_in_4bit_tiles(dev, N, K, gs, B):
    d = cases.make_linear(31 * N + B, N, K, rank=16, fmt="gptq", bits=3, groupsize=gs)
    lin = cases.to_b200_linear(d, dev)
    assert lin._tiled is not None
    assert torch.equal(lin._dequant_gptq().cpu(), O.gptq_tile_fp16(d["qweight_int"], d["scales"], d["zeros"], gs))
    x = cases.make_x(N + B, B, K)
    assert cases.rel_l2(lin(x.to(dev)).cpu(), O.linear_forward(cases.to_oracle_linear(d), x, x_rot_half=True)) <= REL
    d["qweight_int"][0, 0] = 9          # outside 3 bits: the int8 kernel
    lin = cases.to_b200_linear(d, dev)
    assert lin._tiled is None
    assert cases.rel_l2(lin(x.to(dev)).cpu(), O.linear_forward(cases.to_oracle_linear(d), x, x_rot_half=True)) <= REL


@pytest.mark.parametrize("N,K", [(1408, 2048), (72, 256), (19, 132), (64, 64)])
def test_turbo_tiles_bit_exact(dev, N, K):
    from glorcq_b200.tiled import TiledWeight
    d = cases.make_linear(202 + N, N, K, fmt="turbo", with_lora=False)
    tw = TiledWeight.from_turbo(d["packed_indices"].to(dev), d["norms"].to(dev), d["centroids"].to(dev))
    W = tw.dequantize().cpu()
    assert torch.equal(W, O.turbo_tile(d["packed_indices"], d["norms"], d["centroids"], K))


# ---- GLoRCQLinear.forward ------------------------------------------------------------------
LIN = [
    # N, K, rank, fmt, bits, groupsize, sym
    (1408, 2048, 64, "gptq", 2, 128, False),     # expert gate/up projection
    (2048, 1408, 64, "gptq", 2, 128, False),     # expert down projection, 11 groups
    (5632, 2048, 64, "gptq", 2, 128, False),     # shared expert
    (2048, 5632, 64, "gptq", 2, 128, True),
    (2048, 2048, 128, "gptq", 4, 128, False),    # attention projection, 4-bit
    (100, 392, 16, "gptq", 2, 128, False),       # ragged rows, K not a multiple of 128
    (24, 128, 0, "gptq", 2, 128, False),
    (1408, 2048, 64, "turbo", 2, 0, False),
    (2048, 1408, 64, "turbo", 2, 0, False),
    (52, 192, 16, "turbo", 2, 0, False),
]


@pytest.mark.parametrize("B", [1, 2, 5, 8, 13, 16, 33, 70])
@pytest.mark.parametrize("N,K,rank,fmt,bits,gs,sym", LIN)
def test_linear_forward(dev, N, K, rank, fmt, bits, gs, sym, B):
    if B > 16 and N * K > 3_000_000:
        pytest.skip("large batch only on the smaller shapes")
    d = cases.make_linear(7 * N + K + B, N, K, rank=max(rank, 16), fmt=fmt, bits=bits, groupsize=gs or 128, sym=sym,
                          with_lora=rank > 0)
    lin = cases.to_b200_linear(d, dev)
    x = cases.make_x(N + K + 31 * B, B, K)
    y = lin(x.to(dev)).cpu()
    ref = O.linear_forward(cases.to_oracle_linear(d), x, x_rot_half=True)
    assert y.dtype == torch.float16 and y.shape == ref.shape
    assert cases.rel_l2(y, ref) <= REL
    if rank > 0:
        a = (x @ d["U"])
        y2 = lin(x.to(dev), precomputed_xU=a.to(dev)).cpu()
        assert cases.rel_l2(y2, ref) <= REL


def _hostile_rows(B, K, seed):
    """Activation rows that attack the block fixed-point staging of the integer decode path (each 128-channel
    block of a row is scaled by a power of two taken from its largest magnitude): one element 2^10 times the
    rest of its block, a block of fp16 subnormals, a block of zeros, elements at +-60000 beside ordinary
    values, a row of tiny values, and blocks whose sign pattern makes the plain sum cancel."""
    x = cases.make_x(seed, B, K).float()
    nb = K // 128
    for b in range(B):
        x[b, (b % nb) * 128 + 5] *= 1024.0                               # outlier 2^10 x its block
        blk = (b + 1) % nb
        x[b, blk * 128:(blk + 1) * 128] = x[b, blk * 128:(blk + 1) * 128] * 3e-7    # fp16 subnormals
        blk = (b + 2) % nb
        x[b, blk * 128:(blk + 1) * 128] = 0.0
        blk = (b + 3) % nb
        x[b, blk * 128 + 17] = 60000.0
        x[b, blk * 128 + 90] = -60000.0
        blk = (b + 4) % nb
        half = x[b, blk * 128:blk * 128 + 64].clone()
        x[b, blk * 128 + 64:(blk + 1) * 128] = -half                       # sum of the block cancels exactly
    if B > 1:
        x[B - 1] *= 1e-3
    return x.to(torch.float16)


@pytest.mark.parametrize("B", [1, 3, 8])
@pytest.mark.parametrize("N,K,bits", [(1408, 2048, 2), (2048, 1408, 2), (2048, 2048, 4)])
def test_integer_path_hostile_activations(dev, N, K, bits, B):
    """Up to 8 rows of affine codes run on the integer path, which rounds every 128-channel block of x to
    16-bit fixed point relative to the block maximum (exact within 2^-13 of it, absolute error <= 2^-16 of it
    below); the reference multiplies the exact fp16 values.  Outliers, subnormals and near-overflow values
    must still land within the layer bar, rel-L2 <= 1e-3, per row as well as over all rows."""
    d = cases.make_linear(77 * B + N + bits, N, K, rank=64, bits=bits)
    lin = cases.to_b200_linear(d, dev)
    x = _hostile_rows(B, K, 4000 + B + N)
    y = lin(x.to(dev)).cpu()
    ref = O.linear_forward(cases.to_oracle_linear(d), x)
    assert torch.isfinite(ref.float()).all() and torch.isfinite(y.float()).all()
    assert cases.rel_l2(y, ref) <= REL
    for b in range(B):
        assert cases.rel_l2(y[b], ref[b]) <= REL, f"row {b}"


@pytest.mark.parametrize("B", [1, 8, 9, 33, 300])
@pytest.mark.parametrize("N,K,gs", [(2048, 2048, 128), (1000, 768, 64), (72, 14336, 128), (72, 24576, 128)])
def test_3bit_layers_round_their_result_only(dev, N, K, gs, B):
    """3-bit codes are multiplied as the int8 kernel does it: fp16 activations and unrounded (q - z) s, alone and in a group
    of layers, on both sides of 32 rows.  What is left is one fp16 rounding of the result: 2.1e-4 for results that are
    normal values (a uniform error of half a unit over their binades), 2.3e-4 with 8 % for the spread over a few thousand
    results; block fixed point adds 2e-4 and more on these rows, an fp16 weight 2e-4.  (14336: chunks of four rows,
    24576: the general kernel.)"""
    from glorcq_b200 import tiled
    d = cases.make_linear(N + K + B, N, K, bits=3, groupsize=gs, with_lora=False)
    lin = cases.to_b200_linear(d, dev)
    x = (_hostile_rows(B, K, 70 + B) * 0.03125).to(dev)
    q, s, z = (d[k].to(dev).double() for k in ("qweight_int", "scales", "zeros"))
    W = ((q - z.repeat_interleave(gs, 1)[:, :K]) * s.repeat_interleave(gs, 1)[:, :K])
    ref = x.double() @ W.T
    assert float(ref.abs().max()) < 60000
    err = lambda y: float((y.double() - ref).norm() / ref.norm())
    bar = 2.3e-4 * (1 + 1.5 / (N * B) ** 0.5)
    assert err(lin(x)) <= bar
    both = tiled.GroupedLinear([lin._tiled, lin._tiled], None).forward(x)
    assert err(both[0]) <= bar and torch.equal(both[0], both[1])
    assert tiled.debug_error() is None


@pytest.mark.parametrize("N,K,rank,B,int_zeros", [(1408, 2048, 64, 128, True), (2048, 1408, 64, 300, True),
                                                   (100, 392, 16, 200, True), (256, 256, 16, 64, False),
                                                   (24, 128, 0, 40, True), (5632, 2048, 64, 96, True)])
def test_many_rows_tensor_core_path(dev, N, K, rank, B, int_zeros):
    """More than 32 rows of 2-bit affine codes go to the tcgen05 kernel: ragged feature and channel
    counts, token counts that do not fill a tile, non-integer zero points."""
    d = cases.make_linear(11 * N + K + B, N, K, rank=max(rank, 16), with_lora=rank > 0, int_zeros=int_zeros)
    lin = cases.to_b200_linear(d, dev)
    x = cases.make_x(N + 3 * K + B, B, K)
    y = lin(x.to(dev)).cpu()
    ref = O.linear_forward(cases.to_oracle_linear(d), x)
    assert cases.rel_l2(y, ref) <= REL
    from glorcq_b200 import tiled
    assert tiled.debug_error() is None


@pytest.mark.parametrize("N,K,rank,B,int_zeros", [(5632, 2048, 64, 1300, True), (2816, 1024, 16, 2100, False)])
def test_many_rows_more_items_than_sms(dev, N, K, rank, B, int_zeros):
    """Prefill-sized calls whose (token tile, feature tile) items outnumber the SMs: every CTA of the persistent
    tcgen05 kernel takes several items, so the rings run across item boundaries, the accumulator is handed back
    and forth and the results of one item are written while the next one is multiplied.  Last token tile ragged."""
    d = cases.make_linear(5 * N + K + B, N, K, rank=rank, int_zeros=int_zeros)
    lin = cases.to_b200_linear(d, dev)
    x = cases.make_x(N + 7 * K + B, B, K)
    y = lin(x.to(dev)).cpu()
    ref = O.linear_forward(cases.to_oracle_linear(d), x)
    assert cases.rel_l2(y, ref) <= REL
    for b in (0, 255, 256, 1023, 1024, B - 1):
        assert cases.rel_l2(y[b], ref[b]) <= REL, f"row {b}"
    y2 = lin(x.to(dev)).cpu()
    assert torch.equal(y, y2), "two calls in a row differ"
    from glorcq_b200 import tiled
    assert tiled.debug_error() is None


@pytest.mark.parametrize("N,K", [(14336, 4096), (4096, 14336)])
@pytest.mark.parametrize("B", [1, 40])
def test_mixtral_expert_projection_shapes(dev, N, K, B):
    """The largest projections of the benchmark configurations (expert up / down of a Mixtral-8x7B-shaped
    layer): long reductions (112 k blocks) and many row tiles."""
    d = cases.make_linear(3 * N + K + B, N, K, rank=64)
    lin = cases.to_b200_linear(d, dev)
    x = cases.make_x(N + K + B, B, K)
    y = lin(x.to(dev)).cpu()
    ref = O.linear_forward(cases.to_oracle_linear(d), x)
    assert cases.rel_l2(y, ref) <= REL
    from glorcq_b200 import tiled
    assert tiled.debug_error() is None


def test_linear_batch_dims_and_empty(dev):
    d = cases.make_linear(5, 96, 256, rank=16)
    lin = cases.to_b200_linear(d, dev)
    x = cases.make_x(6, 6, 256).reshape(2, 3, 256)
    y = lin(x.to(dev))
    assert y.shape == (2, 3, 96)
    ref = O.linear_forward(cases.to_oracle_linear(d), x)
    assert cases.rel_l2(y.cpu(), ref) <= REL
    y0 = lin(torch.empty(0, 256, dtype=torch.float16, device=dev))
    assert y0.shape == (0, 96)
    torch.cuda.synchronize()


def test_linear_turbo_with_rotation(dev):
    d = cases.make_linear(21, 72, 256, rank=16, fmt="turbo")
    g = torch.Generator().manual_seed(5021)
    q, _ = torch.linalg.qr(torch.randn(256, 256, generator=g))
    d["Pi"] = q.to(torch.float16)
    lin = cases.to_b200_linear(d, dev)
    x = cases.make_x(1021, 4, 256)
    ref = O.linear_forward(cases.to_oracle_linear(d), x, x_rot_half=True)
    assert cases.rel_l2(lin(x.to(dev)).cpu(), ref) <= REL
    xr = (x.float() @ d["Pi"].float().T).half()
    assert cases.rel_l2(lin(x.to(dev), precomputed_x_rot=xr.to(dev)).cpu(), ref) <= REL


@pytest.mark.parametrize("B", [1, 3, 8, 13])
@pytest.mark.parametrize("N,K,rank", [(1408, 2048, 64), (2048, 1408, 64), (52, 192, 16)])
@pytest.mark.parametrize("residue", [0.0, 2e-7])
def test_linear_turbo_symmetric_codebook(dev, N, K, rank, B, residue):
    """A codebook (-a, -b, b, a), the shape a Lloyd-Max fit of a symmetric density gives (exactly, or up to the
    residue of the fit's last iteration): up to 8 rows take the integer path with two integer products per
    block; the sorted random codebooks of the other cases take its three-product form."""
    d = cases.make_linear(900 + N + B, N, K, rank=rank, fmt="turbo")
    c = torch.tensor([-1.51, -0.4528, 0.4528, 1.51], dtype=torch.float64) / K ** 0.5
    c[3] += residue * c[3]
    d["centroids"] = c.float()
    lin = cases.to_b200_linear(d, dev)
    x = cases.make_x(901 + B, B, K)
    ref = O.linear_forward(cases.to_oracle_linear(d), x, x_rot_half=True)
    assert cases.rel_l2(lin(x.to(dev)).cpu(), ref) <= REL


def test_shared_u_is_tiled_once(dev):
    from glorcq_b200 import tiled
    blk = cases.make_moe(77, 256, 128, 4, 2, rank=16, experts_per_cluster=2)
    shared = {}
    lins = [cases.to_b200_linear(ex["gate_proj"], dev, shared) for ex in blk["experts"]]
    assert lins[0]._ut is lins[1]._ut and lins[2]._ut is lins[3]._ut and lins[0]._ut is not lins[2]._ut
    assert lins[0].U.data_ptr() == lins[1].U.data_ptr()


def test_against_golden(dev, golden):
    from tests.golden.make_golden import LINEAR_CASES
    for name, kw, B in LINEAR_CASES:
        d = cases.make_linear(**kw)
        if d["fmt"] == "turbo":
            gen = torch.Generator().manual_seed(kw["seed"] + 5000)
            q, _ = torch.linalg.qr(torch.randn(kw["K"], kw["K"], generator=gen))
            d["Pi"] = q.to(torch.float16)
        lin = cases.to_b200_linear(d, dev)
        x = cases.make_x(kw["seed"] + 1000, B, kw["K"])
        y = lin(x.to(dev)).cpu()
        assert cases.rel_l2(y, golden["linear"][name]["y"]) <= REL, name


# ---- drop-ins for the reference's native modules ---------------------------------------------
@pytest.mark.parametrize("B,N,K", [(1, 1408, 2048), (4, 2048, 1408), (5, 1408, 2048), (16, 4096, 4096),
                                   (32, 512, 14336), (1, 64, 64), (3, 30, 36), (1, 2048, 5632), (8, 5632, 2048)])
def test_turbo_dropin(dev, B, N, K):
    import glorcq_b200.kernels as GK
    g = torch.Generator().manual_seed(B * 1000 + N + K)
    packed = torch.randint(0, 256, (N, K // 4), generator=g, dtype=torch.int32).to(torch.uint8)
    norms = torch.randn(N, generator=g).abs() + 0.1
    centroids = torch.randn(4, generator=g)
    x = torch.randn(B, K, generator=g).half()
    y = GK.turbo_dequant_matmul_fused(None, packed.to(dev), norms.to(dev), None, centroids.to(dev), 2, K,
                                      precomputed_x_rot=x.to(dev))
    ref = O.turbo_matmul(x, packed, norms, centroids)
    assert y.dtype == torch.float16 and tuple(y.shape) == (B, N)
    assert cases.rel_l2(y.cpu(), ref) <= REL


def test_turbo_dropin_empty_batch(dev):
    import glorcq_b200.kernels as GK
    packed = torch.zeros(8, 16, dtype=torch.uint8, device=dev)
    y = GK.turbo_dequant_matmul(torch.empty(0, 64, dtype=torch.float16, device=dev), packed,
                                torch.ones(8, device=dev), torch.ones(4, device=dev))
    assert tuple(y.shape) == (0, 8)
    torch.cuda.synchronize()      # the context stays healthy
    with pytest.raises(RuntimeError):
        GK.turbo_dequant_matmul(torch.empty(1, 64, dtype=torch.float32, device=dev), packed,
                                torch.ones(8, device=dev), torch.ones(4, device=dev))


@pytest.mark.parametrize("E,n_out,K", [(3, 16, 128), (60, 2048, 1408), (5, 100, 256)])
def test_turbo_grouped_dropin(dev, E, n_out, K):
    import glorcq_b200.kernels as GK
    d = cases.make_linear(43 + E, E * n_out, K, fmt="turbo", with_lora=False)
    x = cases.make_x(44 + E, E, K)
    y = GK.turbo_dequant_grouped_gemv_fused(x.to(dev), d["packed_indices"].to(dev), d["norms"].to(dev),
                                            d["centroids"].to(dev), n_out)
    ref = O.turbo_grouped_gemv(x, d["packed_indices"], d["norms"], d["centroids"], n_out)
    assert tuple(y.shape) == (E * n_out,)
    assert cases.rel_l2(y.cpu(), ref) <= REL


@pytest.mark.parametrize("B,N,K,sym,lora", [(1, 1408, 2048, False, False), (4, 2048, 1408, False, True),
                                            (5, 100, 392, True, False), (9, 64, 256, False, True),
                                            (0, 16, 128, False, False)])
def test_gptq_i8_dropin(dev, B, N, K, sym, lora):
    import glorcq_b200.kernels as GK
    d = cases.make_linear(900 + N, N, K, fmt="gptq", with_lora=False, int_zeros=False, sym=sym, signed_codes=True)
    x = cases.make_x(901, B, K, torch.float32)
    lo = cases.make_x(902, B, N, torch.float32) * 0.1 if lora else torch.empty(0)
    q8 = d["qweight_int"].to(torch.int8)
    y = GK.gptq_dequant_matmul(x.to(dev), q8.to(dev), d["scales"].to(dev), d["zeros"].to(dev), 128, sym, lo.to(dev))
    assert y.dtype == torch.float32 and tuple(y.shape) == (B, N)
    if B:
        ref = O.gptq_matmul(x, d["qweight_int"], d["scales"], d["zeros"], 128, sym, lo if lora else None)
        assert cases.rel_l2(y.cpu(), ref) <= 1e-5
        assert float((y.cpu() - ref).abs().max()) < 0.01
        yh = GK.gptq_dequant_matmul_fused(x.half().to(dev), d["qweight_int"].to(dev), d["scales"].to(dev),
                                          d["zeros"].to(dev), 128, sym)
        assert yh.dtype == torch.float16


# ---- routes around the packed formats ----------------------------------------------------------------
@pytest.mark.parametrize("B", [33, 64, 65, 130, 515])
@pytest.mark.parametrize("fmt,bits,gs,N,K,rank", [("gptq", 2, 128, 264, 384, 16), ("gptq", 4, 64, 264, 320, 80), ("gptq", 4, 128, 40, 64, 0),
                                                  ("turbo", 2, 0, 392, 256, 64), ("gptq", 2, 256, 100, 200, 16)])
def test_many_rows_every_format(dev, fmt, bits, gs, N, K, rank, B):
    """The tensor-memory GEMM at the edges of its tiles: token tiles of 64, 128 and 256, ragged features and channels, a
    half-filled last stage, more than one low-rank slice, zero points that are not whole numbers."""
    from glorcq_b200 import tiled
    d = cases.make_linear(N + K + B, N, K, rank=max(rank, 16), fmt=fmt, bits=bits, groupsize=gs or 128, with_lora=rank > 0,
                          int_zeros=B != 65)
    x = cases.make_x(N + B, B, K)
    y = cases.to_b200_linear(d, dev)(x.to(dev)).cpu()
    assert cases.rel_l2(y, O.linear_forward(cases.to_oracle_linear(d), x, x_rot_half=True)) <= REL
    assert tiled.debug_error() is None


@pytest.mark.parametrize("B", [1, 5, 8, 13])
@pytest.mark.parametrize("fmt,bits,N,K", [("gptq", 2, 72, 14336), ("gptq", 4, 4096, 4096), ("turbo", 2, 1000, 8192), ("gptq", 2, 4096, 24576)])
def test_long_reductions(dev, fmt, bits, N, K, B):
    """Rows too long for two CTAs' copies of them: one CTA of eight or sixteen warps, or the general kernel."""
    from glorcq_b200 import tiled
    if N * K > 20_000_000 and B > 5:
        pytest.skip("the longest rows on few of them")
    d = cases.make_linear(N + K, N, K, rank=16, fmt=fmt, bits=bits)
    lin = cases.to_b200_linear(d, dev)
    x = cases.make_x(K + B, B, K)
    y = lin(x.to(dev))
    assert cases.rel_l2(y.cpu(), O.linear_forward(cases.to_oracle_linear(d), x, x_rot_half=True)) <= REL
    for _ in range(3):
        assert torch.equal(y, lin(x.to(dev)))
    assert tiled.debug_error() is None


@pytest.mark.parametrize("N,K", [(64, 2048), (192, 4096), (8, 264), (72, 64), (512, 1408), (520, 256)])
def test_dense_few_columns(dev, N, K):
    """x . W^T with few columns on both sides of 32 rows: row tiles of 32 and 64, column slices of 64."""
    from glorcq_b200 import tiled
    W = torch.randn(N, K, generator=torch.Generator().manual_seed(N + K)).half()
    tw = tiled.TiledWeight.from_dense(W.to(dev))
    for B in (9, 32, 33, 333, 5000):
        x = cases.make_x(B + K, B, K)
        y = tiled.dense_matmul(tw, x.to(dev))
        assert cases.rel_l2(y.cpu(), x.float() @ W.float().T) <= REL, B
        assert torch.equal(y, tiled.dense_matmul(tw, x.to(dev))), B
        off = torch.empty(B * K + 1, dtype=torch.float16, device=dev)[1:].view(B, K).copy_(x)       # rows off 16-byte boundaries
        assert torch.equal(y, tiled.dense_matmul(tw, off)), B
    assert tiled.debug_error() is None


def test_dense_weight_route_dtype_and_reference_op_names(dev):
    """Pre-dequantised weights (a checkpoint's ``weight_quant`` records and the legacy load_turbo_predequant)
    run dense through the fp16 kernels with the low-rank term; a bf16 / fp32 input gets its own dtype back;
    the reference's custom-op names ``torch.ops.glorcq.*`` bind to this package's kernels."""
    from glorcq_b200.quantized_linear import GLoRCQLinear
    import glorcq_b200.kernels as GK
    g = torch.Generator().manual_seed(77)
    N, K, r = 96, 256, 16
    W = (torch.randn(N, K, generator=g) * 0.05).half()
    U = (torch.randn(K, r, generator=g) * 0.01).half()
    SV = (torch.randn(N, r, generator=g) * 0.01).half()
    x = cases.make_x(78, 5, K)
    ref = (x.float() @ W.float().T + (x.float() @ U.float()) @ SV.float().T)
    lin = GLoRCQLinear(K, N)
    lin.load_dense(W, device=dev)
    lin.load_sv(U.to(dev), SV, device=dev)
    y = lin(x.to(dev))
    assert y.dtype == torch.float16 and cases.rel_l2(y.cpu(), ref) <= REL
    for dt in (torch.bfloat16, torch.float32):
        assert lin(x.to(dev).to(dt)).dtype == dt
    d = cases.make_linear(79, N, K, rank=r)
    assert cases.to_b200_linear(d, dev)(x.to(dev).float()).dtype == torch.float32

    class _Quantizer:                      # stands in for the third-party quantizer object
        def dequantize(self, q):
            assert q.bits == 2 and q.indices.shape == (N, K // 4)
            return W.to(q.indices.device)
    lin2 = GLoRCQLinear(K, N)
    lin2.load_turbo_predequant({"packed_indices": torch.zeros(N, K // 4, dtype=torch.uint8), "norms": torch.ones(N),
                                "bits": 2, "dim": K}, _Quantizer(), device=dev)
    assert lin2.quant_type == "turbo" and cases.rel_l2(lin2(x.to(dev)).cpu(), x.float() @ W.float().T) <= REL

    t = cases.make_linear(80, 72, 256, fmt="turbo", with_lora=False)
    y1 = torch.ops.glorcq.turbo_dequant_matmul(x.to(dev), t["packed_indices"].to(dev), t["norms"].to(dev), t["centroids"].to(dev))
    assert cases.rel_l2(y1.cpu(), O.turbo_matmul(x, t["packed_indices"], t["norms"], t["centroids"])) <= REL
    q = cases.make_linear(81, 64, 256, fmt="gptq", with_lora=False, signed_codes=True)
    q32 = q["qweight_int"].to(dev)
    y2 = torch.ops.glorcq.gptq_dequant_matmul(x.float().to(dev), q32.to(torch.int8), q["scales"].to(dev), q["zeros"].to(dev), 128,
                                              False, torch.empty(0, device=dev))
    assert cases.rel_l2(y2.cpu(), O.gptq_matmul(x.float(), q["qweight_int"], q["scales"], q["zeros"], 128, False, None)) <= 1e-5
    # the int8 copy of int32 codes is made once per tensor, and again after the tensor changed
    a8 = GK._int8_codes(q32)
    assert GK._int8_codes(q32) is a8
    q32 += 0
    assert GK._int8_codes(q32) is not a8


# ---- threads ------------------------------------------------------------------------------------------
def test_launches_run_without_the_interpreter_lock(dev):
    """The library's entry points are replaced by PyGILState_Check: 0, a success, when the calling thread does not
    hold the interpreter lock, 1, an unknown status, when it does.  Each is reached by one of the calls: replaced by
    Py_IsInitialized, which is 1, one of them fails."""
    import ctypes as C
    from glorcq_b200 import _lib, tiled
    from glorcq_b200.kernels import gptq_dequant_matmul, turbo_dequant_grouped_gemv, turbo_dequant_matmul
    lin = cases.to_b200_linear(cases.make_linear(3, 64, 128, rank=16), dev)
    group = tiled.GroupedLinear([lin._tiled] * 2, [lin._ut] * 2)
    blk = cases.to_b200_moe(cases.make_moe(5, 128, 64, 4, 2, rank=16, experts_per_cluster=2), dev)
    x = cases.make_x(4, 2, 128).to(dev)
    blk(x.view(1, 2, 128))
    q, n, c = torch.zeros(16, 32, dtype=torch.uint8, device=dev), torch.ones(16, device=dev), torch.ones(4, device=dev)
    s = torch.ones(16, 1, dtype=torch.float16, device=dev)
    plain, signs = tiled.GroupedLinear([lin._tiled] * 2, None), torch.ones(128, device=dev)
    calls = [lambda: lin(x), lambda: group.forward(x), lambda: plain.forward(x), lambda: tiled.linear_forward(lin._tiled, x, lin._ut, signs=signs),
             lambda: blk(x.view(1, 2, 128)), lambda: turbo_dequant_matmul(x, q, n, c),
             lambda: turbo_dequant_grouped_gemv(x, q, n, c, 8), lambda: _lib.native().add_rmsnorm(x, x, s[:1].expand(1, 128).contiguous(), 1e-6),
             lambda: gptq_dequant_matmul(x.float(), torch.zeros(16, 128, dtype=torch.int8, device=dev), s, s, 128, False, torch.empty(0, device=dev))]
    for f in calls:
        f()
    nat = _lib.native()
    real = {e: C.cast(getattr(_lib.lib(), e), C.c_void_p).value for e in nat.names()}
    probe = C.cast(C.pythonapi.PyGILState_Check, C.c_void_p).value
    fails = C.cast(C.pythonapi.Py_IsInitialized, C.c_void_p).value
    launches = [e for e in nat.names() if not e.endswith(("_bytes", "_counters")) and e not in ("glq_status_string", "glq_last_cuda_error")]

    def failing():
        out = 0
        for f in calls:
            try:
                f()
            except RuntimeError:
                out += 1
        return out
    try:
        nat.bind({**real, **{e: probe for e in launches}})
        for f in calls:
            f()
        for e in launches:
            nat.bind({**real, **{o: probe for o in launches}, e: fails})
            assert failing() > 0, e
    finally:
        nat.bind(real)


def test_threads_on_one_stream_share_its_scratch(dev):
    """x.U and the product's operands lie in the stream's scratch: calls of several threads must not mix there."""
    import threading
    work = []
    for i, B in enumerate((1, 40, 7, 300)):
        lin = cases.to_b200_linear(cases.make_linear(50 + i, 256, 512, rank=32), dev)
        x = cases.make_x(60 + i, B, 512).to(dev)
        work.append((lin, x, lin(x)))
    wrong = []

    def many(lin, x, ref):
        for _ in range(100):
            if not torch.equal(lin(x), ref):
                wrong.append(x.shape)
    threads = [threading.Thread(target=many, args=w) for w in work]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong


def test_scratch_of_a_captured_call_outlives_a_larger_call(dev):
    """The graph writes x.U and reads it back in the scratch it was captured with."""
    from glorcq_b200 import _lib
    small, large = (cases.to_b200_linear(cases.make_linear(90 + i, 256, K, rank=32), dev) for i, K in enumerate((512, 4096)))
    x, xl = cases.make_x(92, 4, 512).to(dev), cases.make_x(93, 1000, 4096).to(dev)
    ref = small(x)
    st, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    _lib.native().clear_workspaces()
    with torch.cuda.stream(st):
        small(x)
        st.synchronize()
        with torch.cuda.graph(graph, stream=st):
            y = small(x)
        before = _lib.native().workspace(0, 0, 0)[0].numel()
        large(xl)
        assert _lib.native().workspace(0, 0, 0)[0].numel() > before
        others = [torch.full((before // 4,), 7, dtype=torch.int32, device=dev) for _ in range(16)]
        graph.replay()
    st.synchronize()
    assert torch.equal(y, ref)
    assert all(bool((t == 7).all()) for t in others)


@pytest.mark.parametrize("B", [1, 4, 5, 8])
@pytest.mark.parametrize("fmt,bits,N,K,rank,one_launch", [
    ("gptq", 2, 1408, 2048, 64, 8), ("gptq", 4, 520, 896, 16, 8), ("gptq", 3, 40, 192, 128, 8), ("turbo", 2, 1000, 8192, 80, 8),
    # (8 rows of 4096 channels leave an SM one CTA, and the product has one for every SM; 8 of 14336 are the general kernel's; the
    # product of 14336 features has a CTA for every slot)
    ("gptq", 4, 4096, 4096, 64, 4), ("gptq", 2, 72, 14336, 32, 4), ("gptq", 2, 14336, 4096, 64, 0)])
def test_low_rank_operand_in_the_products_launch(dev, fmt, bits, N, K, rank, one_launch, B):
    """x.U computed by the first blocks of the product's launch (up to `one_launch` rows, by a launch of its own above) gives the bits of
    x.U computed alone and handed in, call after call, and leaves the arrival counters at zero."""
    from glorcq_b200 import _lib, tiled
    lin = cases.to_b200_linear(cases.make_linear(N + K + B, N, K, rank=rank, fmt=fmt, bits=bits), dev)
    # (two inputs in turn: the scratch holds the other one's x.U when a call begins)
    xs = [cases.make_x(B + N + i, B, K).to(dev) for i in range(2)]
    refs = [tiled.linear_forward(lin._tiled, x, a=tiled.dense_matmul(lin._ut, x)) for x in xs]
    for i in range(6):
        assert torch.equal(tiled.linear_forward(lin._tiled, xs[i % 2], lin._ut), refs[i % 2])
    torch.cuda.synchronize()
    assert not bool(_lib.native().workspace(0, 0, 0)[1].any()) and tiled.debug_error() is None
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        for x in xs:
            tiled.linear_forward(lin._tiled, x, lin._ut)
    names = [n for edge in _programmatic_edges(graph) for n in edge]
    assert all("stream_pair_kernel" in n for n in names) if B <= one_launch else not any("stream_pair_kernel" in n for n in names), names
    assert names


@pytest.mark.parametrize("B", [1, 5, 8, 9])
@pytest.mark.parametrize("P,fmt,bits,N,K,rank", [(2, "gptq", 2, 520, 896, 16), (3, "gptq", 4, 2048, 2048, 64), (3, "gptq", 3, 40, 192, 80),
                                                 (2, "turbo", 2, 1000, 2048, 64)])
def test_group_with_low_rank_factors(dev, P, fmt, bits, N, K, rank, B):
    """Layers of their own weights and factors, several in a launch (up to 8 rows with their x.U in its first blocks): the results of the layers
    one by one within the rounding of two fp16 results, the same bits call after call, and zero arrival counters."""
    from glorcq_b200 import _lib, tiled
    lins = [cases.to_b200_linear(cases.make_linear(8000 + N + B + i, N, K, rank=rank, fmt=fmt, bits=bits), dev) for i in range(P)]
    group = tiled.GroupedLinear([m._tiled for m in lins], [m._ut for m in lins])
    xs = [cases.make_x(8100 + N + i, B, K).to(dev) for i in range(2)]
    refs = [torch.stack([m(x) for m in lins]) for x in xs]
    got = [group.forward(xs[i % 2]) for i in range(6)]
    for i, y in enumerate(got):
        assert torch.equal(y, got[i % 2])
        assert cases.rel_l2(y.cpu(), refs[i % 2].cpu()) <= REL
    torch.cuda.synchronize()
    assert not bool(_lib.native().workspace(0, 0, 0)[1].any()) and tiled.debug_error() is None


@pytest.mark.parametrize("rows", [1, 8, 33, 300])
def test_layer_captured_behind_an_event(dev, rows):
    """A layer's first launch may start beside the launch ahead of it; behind an event of another stream, in a graph and
    outside, it still sees what that stream wrote."""
    d = cases.make_linear(4100 + rows, 256, 512, rank=32)
    lin = cases.to_b200_linear(d, dev)
    x = cases.make_x(4200 + rows, rows, 512).to(dev)
    side = torch.cuda.Stream()

    def step():
        main = torch.cuda.current_stream()
        big = torch.ones(1 << 24, device=dev).cumsum(0)          # (the writer of the layer's input starts late)
        x2 = x + x + 0 * big[0].half()
        side.wait_stream(main)
        with torch.cuda.stream(side):
            y = lin(x2)
        main.wait_stream(side)
        return y + 0
    want = lin(x + x)
    for _ in range(2):
        assert torch.equal(step(), want)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        y = step()
    for _ in range(3):
        y.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(y, want)
    from glorcq_b200 import tiled
    assert tiled.debug_error() is None


def test_threads_on_streams_of_their_own(dev):
    """Calls of one kernel that need more and less shared memory, from threads on streams of their own."""
    import threading
    work = []
    for i, (B, K) in enumerate(((4, 512), (8, 4096), (6, 2048), (3, 5632))):
        lin = cases.to_b200_linear(cases.make_linear(150 + i, 256, K, rank=32), dev)
        xs = [cases.make_x(160 + i + 10 * j, B, K).to(dev) for j in range(2)]
        work.append((lin, xs, torch.cuda.Stream()))
    got, errors = {}, []
    start = threading.Barrier(len(work))

    def many(i, lin, xs, st):
        try:
            start.wait()
            with torch.cuda.stream(st):
                got[i] = [lin(xs[j % 2]) for j in range(50)]
        except Exception as e:      # noqa: BLE001
            errors.append(e)
    torch.cuda.synchronize()
    threads = [threading.Thread(target=many, args=(i, *w)) for i, w in enumerate(work)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not errors
    for i, (lin, xs, _) in enumerate(work):
        refs = [lin(x) for x in xs]
        assert all(torch.equal(y, refs[j % 2]) for j, y in enumerate(got[i]))


def _programmatic_edges(graph):
    """[(kernel ahead, kernel started beside it)] of a captured graph of kernels"""
    import ctypes as C
    cu, g, n = C.CDLL("libcuda.so.1"), C.c_void_p(graph.raw_cuda_graph()), C.c_size_t(0)
    assert cu.cuGraphGetEdges_v2(g, None, None, None, C.byref(n)) == 0
    src, dst, data = (C.c_void_p * n.value)(), (C.c_void_p * n.value)(), (C.c_ubyte * (8 * n.value))()      # data: ports, then the type
    assert cu.cuGraphGetEdges_v2(g, src, dst, data, C.byref(n)) == 0

    def name(node):
        p, s = (C.c_void_p * 16)(), C.c_char_p()             # CUDA_KERNEL_NODE_PARAMS_v2: func, seven ints, two pointers, kern
        assert cu.cuGraphKernelNodeGetParams_v2(C.c_void_p(node), p) == 0
        rc = cu.cuFuncGetName(C.byref(s), C.c_void_p(p[0])) if p[0] else cu.cuKernelGetName(C.byref(s), C.c_void_p(p[7]))
        assert rc == 0
        return s.value.decode()
    return [(name(a), name(b)) for a, b, kind in zip(src, dst, data[2::8]) if kind == 1]


@pytest.mark.parametrize("fmt,bits", [("gptq", 2), ("gptq", 4), ("gptq", 3), ("turbo", 2)])
@pytest.mark.parametrize("B", [1, 8])
def test_layer_directly_behind_its_packing(dev, fmt, bits, B):
    """A layer's launch reads weights while the launch ahead of it still runs: that is never the kernel which packs them.  Without the
    caller's word in the descriptor it waits first."""
    from glorcq_b200 import _lib, tiled
    lin = cases.to_b200_linear(cases.make_linear(7100 + bits + B, 1408, 2048, rank=64, fmt=fmt, bits=bits), dev)
    x = cases.make_x(7200 + B, B, 2048).to(dev)
    pool = [(cases.make_x(7300 + i, 2048, 64).to(dev) * 0.01, cases.make_x(7400 + i, 1408, 64).to(dev) * 0.01) for i in range(2)]
    refs = []
    for U, SV in pool:
        lin.load_sv(U, SV)
        torch.cuda.synchronize()
        refs.append(tiled.linear_forward(lin._tiled, x, a=tiled.dense_matmul(lin._ut, x)))
    assert not torch.equal(*refs)
    for i in range(20):                                 # the buffer of SV is packed anew, U^T comes from the pool
        lin.load_sv(*pool[i % 2])
        assert torch.equal(tiled.linear_forward(lin._tiled, x, lin._ut), refs[i % 2]), i
    for i in range(20):                                 # and U^T packed last
        lin.load_sv(pool[i % 2][0].clone(), pool[i % 2][1])
        assert torch.equal(tiled.linear_forward(lin._tiled, x, lin._ut), refs[i % 2]), i
    torch.cuda.synchronize()
    for word in (_lib.WEIGHT_SETTLED, 0):
        graph = torch.cuda.CUDAGraph(keep_graph=True)
        with torch.cuda.graph(graph):
            lin._tiled.put_sv(0, pool[1][1])
            lin._tiled._native = None
            lin._tiled.desc.reserved = word
            y = [tiled.linear_forward(lin._tiled, x, lin._ut) for _ in range(2)]
        edges = _programmatic_edges(graph)
        assert ["pair" in b for _, b in edges] == [True, True] and not any("pack" in a for a, _ in edges), edges
        lin._tiled.put_sv(0, pool[0][1])
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(y[0], refs[1]) and torch.equal(y[1], refs[1])
    assert tiled.debug_error() is None


@pytest.mark.parametrize("bits,N,K,rank,B", [(2, 32, 128, 16, 1), (2, 1408, 2048, 64, 1), (4, 2048, 2048, 128, 5), (3, 520, 896, 80, 8)])
def test_counters_of_a_layer_in_one_launch(dev, bits, N, K, rank, B):
    """The row tiles of x.U are counted in and taken off again, whether the product's wait for them ran out or not (a counter that
    starts two short stands for tiles that come late: cleared, it would end two too high); the call after it is right."""
    import ctypes as C
    from glorcq_b200 import _lib, tiled
    L = _lib.lib()
    lin = cases.to_b200_linear(cases.make_linear(7500 + N, N, K, rank=rank, bits=bits), dev)
    t = lin._tiled
    x, y = cases.make_x(7600 + N, B, K).to(dev), torch.empty(B, N, dtype=torch.float16, device=dev)
    ref = tiled.linear_forward(t, x, a=tiled.dense_matmul(lin._ut, x))
    n_bytes = L.glq_linear_workspace_bytes(t.fmt, t.group_size, C.byref(t.desc), B)
    n_ctr = L.glq_linear_counters(t.fmt, t.group_size, C.byref(t.desc), B)
    ws, ctr = torch.empty(n_bytes, dtype=torch.uint8, device=dev), torch.zeros(n_ctr, dtype=torch.int32, device=dev)

    def call():
        _lib.check(L.glq_linear_forward(t.fmt, t.group_size, C.byref(t.desc), lin._ut.codes.data_ptr(), x.data_ptr(), K, None, y.data_ptr(), N, B,
                                        ws.data_ptr(), n_bytes, ctr.data_ptr(), n_ctr, tiled._stream_ptr(dev)), "linear_forward")
    call()
    assert torch.equal(y, ref) and not ctr.any() and tiled.debug_error() is None
    ctr[-2] = -2                                        # (the last two are those of x.U and its product)
    call()
    assert tiled.debug_error()[0] == 112
    assert ctr[-2] == -2 and not ctr[:-2].any() and ctr[-1] == 0
    ctr[-2] += 2                                        # the two that were late
    y.zero_()
    call()
    assert torch.equal(y, ref) and not ctr.any() and tiled.debug_error() is None


def test_pair_of_a_weight_without_its_low_rank_factor(dev):
    """Nobody waits for x.U then: it is computed all the same, and the counters are zero once the launch is complete."""
    import ctypes as C
    from glorcq_b200 import _lib, tiled
    lin = cases.to_b200_linear(cases.make_linear(7701, 64, 4096, rank=64), dev)
    x = cases.make_x(7702, 3, 4096).to(dev)
    t, a, y = lin._tiled, torch.empty(3, 64, dtype=torch.float16, device=dev), torch.empty(3, 64, dtype=torch.float16, device=dev)
    ws, ctr = torch.empty(1 << 20, dtype=torch.uint8, device=dev), torch.zeros(1 << 12, dtype=torch.int32, device=dev)
    u, m = _lib.MMArgs(), _lib.MMArgs()
    for g, out, n in ((u, a, 64), (m, y, 64)):
        g.n_problems, g.max_rows, g.rows_stride, g.N, g.K = 1, 3, 3, n, 4096
        g.x, g.ldx, g.y, g.ldy = x.data_ptr(), 4096, out.data_ptr(), n
        g.workspace, g.workspace_bytes, g.counters, g.n_counters = ws.data_ptr(), ws.numel(), ctr.data_ptr(), ctr.numel()
    u.fmt, u.w = _lib.FMT_F16, lin._ut.desc
    m.fmt, m.group_size, m.rank, m.a0, m.lda, m.flags = t.fmt, t.group_size, 64, a.data_ptr(), 64, 1
    m.w = _lib.Weight.from_buffer_copy(bytes(t.desc))
    m.w.sv = None
    want, a_want = tiled.linear_forward(t, x, a=torch.zeros_like(a)), tiled.dense_matmul(lin._ut, x)
    for _ in range(20):
        _lib.check(_lib.lib().glq_grouped_matmul_pair(C.byref(u), C.byref(m), tiled._stream_ptr(dev)), "pair")
        assert torch.equal(y, want) and torch.equal(a, a_want) and not ctr.any()
