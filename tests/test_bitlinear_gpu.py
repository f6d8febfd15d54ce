"""GPU parity of the BitLinear path against the CPU oracle, through the C ABI.

Tiers: exact-int (int32 accumulators bitwise equal to the oracle's, which equals the
reference CPU kernel on integer-valued inputs, kernels/cpu.rs:73-124); f32 outputs of the
quantised pipeline within 1e-3 relative (they are expected to be bit-identical); bf16
outputs within one bf16 ulp of the rounded oracle."""
import numpy as np
import pytest

from gpu_util import load_bt, ternary_packed

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

REL_TOL = 1e-3  # stated tolerance for floating-point outputs


@pytest.fixture(scope="module")
def bt():
    if not torch.cuda.is_available():
        pytest.fail("GPU tests need a CUDA device")
    return load_bt()


SHAPES = [  # (m, n, k)
    (1, 16, 256), (1, 64, 64), (1, 256, 688), (3, 100, 4), (1, 17, 36), (8, 2048, 2048),
    (2, 688, 256), (1, 4096, 4096), (5, 1024, 4096), (7, 48, 14336), (17, 64, 512), (33, 32, 256),
    # product kernel for up to 8 tokens: 16 KB ring stages (8 tokens of a long K leave no room for
    # 32 KB ones), an odd number of row tiles per CTA, and more row tiles per CTA than the ring has
    # slots and than there are accumulate buffers (slots and buffers are reused)
    (8, 160, 14336), (1, 7120, 4096), (1, 41000, 512), (3, 41000, 512),
    # one rank's slices of the 8B projections under 8-way tensor parallelism
    (1, 4096, 512), (1, 4096, 1792), (1, 768, 4096), (2, 3584, 4096),
]


@pytest.mark.parametrize("m,n,k", SHAPES)
def test_int32_accumulators_bit_exact(bt, oracle, m, n, k):
    rng = np.random.default_rng(1000 + m + n + k)
    packed = ternary_packed(rng, n, k, p_code3=0.02)
    q = rng.integers(-127, 128, size=(m, k), dtype=np.int8)
    lin = bt.BitLinear.from_packed(packed, [1.0], n, k)
    acc = lin.forward_q(torch.from_numpy(q).cuda()).cpu().numpy()
    ref = oracle.bitlinear_i32(q, packed, n)
    assert np.array_equal(acc, ref)
    # the reference f32 kernel on the same integer-valued inputs gives the same integers
    ref_f = oracle.bitlinear_f32(q.astype(np.float32), packed, n, 1.0)
    assert np.array_equal(acc.astype(np.float32), ref_f)


def test_saturation_rows(bt, oracle):
    # all +1 / all -1 weights against +-127 activations: the largest accumulators possible
    n, k = 32, 14336
    codes = np.zeros((n, k // 4), np.uint8)
    codes[0::2] = 0x55  # +1
    codes[1::2] = 0xAA  # -1
    q = np.full((2, k), 127, np.int8)
    q[1] = -127
    lin = bt.BitLinear.from_packed(codes, [1.0], n, k)
    acc = lin.forward_q(torch.from_numpy(q).cuda()).cpu().numpy()
    assert acc[0, 0] == 127 * k and acc[0, 1] == -127 * k and acc[1, 0] == -127 * k
    assert np.array_equal(acc, oracle.bitlinear_i32(q, codes, n))


def test_config1_forward_f32(bt, oracle):
    # 2048x2048 ternary weight, scale = mean|N(0,0.02)|, 8 tokens x 2048 ~ N(0,1)
    rng = np.random.default_rng(1234)
    n = k = 2048
    packed = ternary_packed(rng, n, k)
    scale = float(np.abs(np.random.default_rng(99).normal(0, 0.02, n * k)).mean() + 1e-6)
    x = np.random.default_rng(1235).normal(0, 1, (8, k)).astype(np.float32)
    lin = bt.BitLinear.from_packed(packed, [scale], n, k)
    y = lin.forward(torch.from_numpy(x).cuda()).cpu().numpy()
    ref = oracle.bitlinear_q(x, packed, [scale], n)
    assert np.abs(y - ref).max() <= REL_TOL * np.abs(ref).max()
    assert np.array_equal(y, ref)  # same operations in the same order
    # host-buffer entry point gives the same numbers
    assert np.array_equal(lin.forward_host(x), y)
    # informational: distance to the reference's un-quantised f32 kernel
    full = oracle.bitlinear_f32(x, packed, n, scale)
    assert np.abs(y - full).max() <= 0.05 * np.abs(full).max()


def test_act_quant_matches_oracle(bt, oracle):
    rng = np.random.default_rng(7)
    x = rng.normal(0, 1, (5, 688)).astype(np.float32)
    x[3] = 0
    q, s, qs = bt.act_quant(torch.from_numpy(x).cuda())
    q0, s0, qs0 = oracle.act_quant(x)
    assert np.array_equal(q.cpu().numpy(), q0)
    assert np.array_equal(s.cpu().numpy(), s0)
    assert np.array_equal(qs.cpu().numpy(), qs0)


def test_pack_then_forward_like_reference_layer(bt, oracle):
    # BitLinear::load + precompute_packed + forward on a rank-3 input
    rng = np.random.default_rng(21)
    n, k = 96, 128
    w = rng.normal(0, 0.02, (n, k)).astype(np.float32)
    lin = bt.BitLinear.load(k, n, w)
    lin.precompute_packed()
    x = rng.normal(0, 1, (2, 3, k)).astype(np.float32)
    y = lin.forward(torch.from_numpy(x).cuda()).cpu().numpy()
    assert y.shape == (2, 3, n)
    p, s = oracle.pack_l1(w)
    ref = oracle.bitlinear_q(x.reshape(6, k), p, [s], n).reshape(2, 3, n)
    assert np.array_equal(y, ref)


def test_multi_basis_converted_layout(bt, oracle):
    rng = np.random.default_rng(31)
    n, k, nb = 80, 320, 3
    bases = rng.integers(-1, 2, size=(nb, n, k)).astype(np.int8)
    packed = oracle.pack_l2(bases)
    scales = np.array([0.02, 0.007, 0.003], np.float32)
    x = rng.normal(0, 1, (4, k)).astype(np.float32)
    lin = bt.BitLinear.from_packed(packed, scales, n, k)
    y = lin.forward(torch.from_numpy(x).cuda()).cpu().numpy()
    ref = oracle.bitlinear_q(x, packed, scales, n, n_bases=nb)
    assert np.abs(y - ref).max() <= REL_TOL * np.abs(ref).max()
    assert np.array_equal(y, ref)
    # and against the reference's dense reconstruction on the quantised activations
    wd = oracle.decode_l2(packed, scales)
    qx, sx, _ = oracle.act_quant(x)
    dense = (qx.astype(np.float32) * sx[:, None]) @ wd.T
    assert np.abs(y - dense).max() <= REL_TOL * np.abs(dense).max()


def test_bf16_in_out(bt, oracle):
    rng = np.random.default_rng(41)
    n, k = 256, 1024
    packed = ternary_packed(rng, n, k)
    x = torch.from_numpy(rng.normal(0, 1, (3, k)).astype(np.float32)).bfloat16()
    lin = bt.BitLinear.from_packed(packed, [0.016], n, k)
    y = lin.forward(x.cuda()).float().cpu().numpy()
    ref = oracle.bitlinear_q(x.float().numpy(), packed, [0.016], n)
    ref_bf16 = torch.from_numpy(ref).bfloat16().float().numpy()
    assert np.array_equal(y, ref_bf16)


def test_shape_error_wording(bt):
    packed = np.zeros((16, 16), np.uint8)
    lin = bt.BitLinear.from_packed(packed, [1.0], 16, 64)
    with pytest.raises(bt.BitTTTError) as ei:
        lin.forward(torch.zeros(2, 32, device="cuda"))
    assert ei.value.status == bt.BT_ERR_SHAPE
    assert "Shape mismatch: Input [2, 32] vs Weight [16, 64]" in ei.value.message  # kernels/cpu.rs:22-30
    with pytest.raises(bt.BitTTTError) as ei:
        bt.BitLinear.from_packed(np.zeros(16 * 4, np.uint8), [1.0], 16, 18)
    assert ei.value.status == bt.BT_ERR_ALIGN
    assert lin.forward(torch.zeros(0, 64, device="cuda")).shape == (0, 16)  # empty input
    assert bt.lib().bt_device_check(0) == 0


@pytest.mark.parametrize("m,n,k", [(9, 128, 256), (64, 256, 1024), (100, 1000, 688), (300, 2048, 2048), (130, 48, 4096)])
def test_tensor_core_path_many_tokens(bt, oracle, m, n, k):
    # more than 8 tokens go through the tcgen05 kernel; same bits as the oracle pipeline
    rng = np.random.default_rng(m * 7 + n)
    packed = ternary_packed(rng, n, k, p_code3=0.01)
    x = rng.normal(0, 1, (m, k)).astype(np.float32)
    x[m // 2] = 0  # an all-zero token
    lin = bt.BitLinear.from_packed(packed, [0.016], n, k)
    y = lin.forward(torch.from_numpy(x).cuda()).cpu().numpy()
    ref = oracle.bitlinear_q(x, packed, [0.016], n)
    assert np.abs(y - ref).max() <= REL_TOL * np.abs(ref).max()
    assert np.array_equal(y, ref)
    assert bt.lib().bt_device_check(0) == 0


@pytest.mark.parametrize("m,bases,nbytes", [
    (200, 1, 0), (200, 3, 0),              # one pass
    (200, 1, 160 << 10), (130, 3, 300 << 10),  # the padded token blocks do not fit: passes of 128 tokens
    (100, 1, 80 << 10), (90, 2, 190 << 10),    # passes of 64 tokens
    (20, 1, 16 << 10), (9, 3, 0)])         # not even a block: the streaming product; the smallest count above eight
@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_forward_takes_what_the_workspace_holds(bt, oracle, m, bases, nbytes, dtype):
    # more than 8 tokens, single and several bases: the same bits whatever the number of passes
    n, k = 300, 516
    rng = np.random.default_rng(m + bases)
    packed = np.stack([ternary_packed(rng, n, k) for _ in range(bases)], -1)
    scales = np.array([0.5 / 3 ** b for b in range(bases)], np.float32)
    x = torch.from_numpy(rng.normal(0, 1, (m, k)).astype(np.float32)).to(getattr(torch, dtype))
    lin = bt.BitLinear.from_packed(packed, scales, n, k)
    y = lin.forward(x.cuda(), workspace=bt.Workspace(nbytes=nbytes)).cpu()
    ref = torch.from_numpy(oracle.bitlinear_q(x.float().numpy(), packed, scales, n, bases)).to(x.dtype)
    assert torch.equal(y, ref)


@pytest.mark.parametrize("m,k", [(255, 4096), (255, 4100), (256, 516), (257, 4100), (256, 16384), (256, 16388), (592, 4096), (593, 4096)])
@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_row_quantisers(bt, oracle, m, k, dtype):
    # both sides of the row counts and row lengths at which another row kernel is taken; rows of no 16-byte alignment
    # (bf16, 516 and 4100 values), a row of zeros, values that tie between two integers
    n = 48
    rng = np.random.default_rng(m + k)
    packed = ternary_packed(rng, n, k)
    x = rng.normal(0, 1, (m, k)).astype(np.float32)
    x[3], x[m - 1, :5] = 0, [127, 0.5, -0.5, 126.5, -1.5]
    x = torch.from_numpy(x).to(getattr(torch, dtype))
    lin = bt.BitLinear.from_packed(packed, [0.5], n, k)
    y = lin.forward(x.cuda()).cpu()
    ref = torch.from_numpy(oracle.bitlinear_q(x.float().numpy(), packed, [0.5], n)).to(x.dtype)
    assert torch.equal(y, ref)


@pytest.mark.parametrize("m,n,k", [
    (129, 9217, 260),    # the last tile's second half: no rows; one token in the second token block
    (300, 6300, 516),    # token blocks in odd number: a half without tokens
    (2049, 1160, 1028),  # more token blocks than row tiles
    (1030, 9000, 256),   # several tiles of a single 256-input chunk
    (129, 9217, 1796), (300, 6300, 2052), (2049, 1160, 2048), (600, 8300, 1792),  # with pairs, the last one on their near side
])
@pytest.mark.parametrize("dtype,bases", [("float32", 1), ("bfloat16", 1), ("float32", 2), ("bfloat16", 3)])
def test_tensor_core_path_cta_pairs(bt, oracle, m, n, k, dtype, bases):
    # products of tiles of 256 rows x 256 tokens over two CTAs (from 2048 inputs on, rounded up to 256): the oracle's bits
    rng = np.random.default_rng(m + n + bases)
    packed = np.stack([ternary_packed(rng, n, k, p_code3=0.01) for _ in range(bases)], -1)
    scales = np.array([0.5 / 3 ** b for b in range(bases)], np.float32)
    x = torch.from_numpy(rng.normal(0, 1, (m, k)).astype(np.float32)).to(getattr(torch, dtype))
    x[m // 2] = 0
    lin = bt.BitLinear.from_packed(packed, scales, n, k)
    y = lin.forward(x.cuda()).cpu()
    ref = torch.from_numpy(oracle.bitlinear_q(x.float().numpy(), packed, scales, n, bases)).to(x.dtype)
    assert torch.equal(y, ref)
    assert bt.lib().bt_device_check(0) == 0




@pytest.mark.parametrize("m,n,k,bases", [
    (9, 4000, 14336, 1), (64, 512, 8192, 1), (64, 20000, 2048, 1), (40, 1024, 8192, 3),  # inputs cut over clusters, 256-row tiles, several bases
    (130, 1000, 14336, 1), (300, 9217, 4096, 1), (2049, 1160, 8192, 1)])                # 128-row tiles, CTA pairs
def test_products_under_traffic(bt, m, n, k, bases):
    # copies that come late and out of order, because another stream takes the memory: the bits of an idle GPU
    rng = np.random.default_rng(m)
    packed = np.stack([ternary_packed(rng, n, k) for _ in range(bases)], -1)
    lin = bt.BitLinear.from_packed(packed, [0.5 / 3 ** b for b in range(bases)], n, k)
    x = torch.from_numpy(rng.normal(0, 1, (m, k)).astype(np.float32)).cuda()
    ws, want, side = bt.Workspace(nbytes=64 << 20), lin.forward(x), torch.cuda.Stream()
    a, b = torch.empty(2, 1 << 27, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        for _ in range(40):  # 2 ms
            b.copy_(a)
    got = [lin.forward(x, workspace=ws) for _ in range(20)]
    torch.cuda.synchronize()
    assert all(torch.equal(y, want) for y in got)
    assert bt.lib().bt_device_check(0) == 0


@pytest.mark.parametrize("m,n,k,bases", [
    (9, 128, 256, 2), (40, 300, 516, 8),                     # one row tile; eight bases, rows that fill no tile
    (16, 4096, 4096, 3), (33, 1000, 8192, 3), (64, 600, 2048, 2),  # inputs cut over clusters
    (64, 19100, 260, 2)])                                    # more row tiles than SMs
@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_bases_in_one_launch(bt, oracle, m, n, k, bases, dtype):
    # 9 to 64 tokens: the bases of a projection are worked through in one launch and added up in basis order
    rng = np.random.default_rng(m + n)
    packed = np.stack([ternary_packed(rng, n, k) for _ in range(bases)], -1)
    scales = np.array([0.5 / 3 ** b for b in range(bases)], np.float32)
    x = torch.from_numpy(rng.normal(0, 1, (m, k)).astype(np.float32)).to(getattr(torch, dtype))
    lin = bt.BitLinear.from_packed(packed, scales, n, k)
    ref = torch.from_numpy(oracle.bitlinear_q(x.float().numpy(), packed, scales, n, bases)).to(x.dtype)
    for _ in range(2):  # (the second time over an output that is not zero)
        y = lin.forward(x.cuda()).cpu()
        assert torch.equal(y, ref)
    assert bt.lib().bt_device_check(0) == 0


@pytest.mark.parametrize("k", [16, 272, 8192, 16384, 16400, 516])  # the last two stay with the quantiser kernel
@pytest.mark.parametrize("m", [1, 2, 3, 4])  # the last count too
@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_rows_quantised_in_the_product(bt, oracle, m, k, dtype):
    n = 100
    rng = np.random.default_rng(m * k)
    packed = ternary_packed(rng, n, k)
    x = rng.normal(0, 1, (m, k)).astype(np.float32)
    x[0, :5] = [127, 0.5, -0.5, 126.5, -1.5]
    if m > 1:
        x[1] = 0
    if m > 2:
        x[2] *= 1e-39  # 127 / max|x| overflows: every value saturates
    x = torch.from_numpy(x).to(getattr(torch, dtype))
    if m > 2:  # (but for zeros, whose product with infinity is no number: the oracle's conversion of it to an integer is not defined)
        x[2][x[2] == 0] = 2.0 ** -130
    lin = bt.BitLinear.from_packed(packed, [0.5], n, k)
    ref = torch.from_numpy(oracle.bitlinear_q(x.float().numpy(), packed, [0.5], n)).to(x.dtype)
    assert torch.equal(lin.forward(x.cuda()).cpu(), ref)
    apart = torch.empty(m * k + 1, dtype=x.dtype, device="cuda")[1:].view(m, k).copy_(x)  # rows that start on no 16-byte boundary
    assert torch.equal(lin.forward(apart).cpu(), ref)
    # values that are no numbers, as the quantiser kernel has them (more tokens than the product quantises itself)
    tiny = torch.cat([torch.zeros(1, k // 2), torch.full((1, k // 2), 2.0 ** -130)], 1).to(x.dtype)
    assert torch.equal(lin.forward(tiny.cuda()), lin.forward(tiny.expand(4, k).contiguous().cuda())[:1])
    x[0, 3], x[0, k // 2] = float("nan"), float("inf")
    many = x[:1].expand(4, k).contiguous().cuda()
    assert torch.equal(lin.forward(x[:1].cuda()).nan_to_num(7.0), lin.forward(many)[:1].nan_to_num(7.0))
    assert bt.lib().bt_device_check(0) == 0


@pytest.mark.parametrize("m", [1, 2, 3, 4, 9, 130])  # on both sides of where the product quantises its rows itself, and of the tensor-core product
@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_in_place(bt, m, dtype):
    # outputs over the inputs, and over a part of them, through the C entry: what the call with outputs of their own gives
    n = 8192  # more row tiles than CTAs that run at once: the last outputs are stored long after the first
    rng = np.random.default_rng(m)
    lin = bt.BitLinear.from_packed(ternary_packed(rng, n, n), [0.5], n, n)
    x = torch.from_numpy(rng.normal(0, 1, (m, n)).astype(np.float32)).to(getattr(torch, dtype)).cuda()
    want, code = lin.forward(x), 0 if dtype == "float32" else 1
    for shift in (0, 16, n // 2):  # y begins so many values into x
        if shift and m > 8:
            continue  # (every row has been read only up to a pass of the tensor-core product)
        for _ in range(4):
            buf = torch.empty(m * n + shift, dtype=x.dtype, device="cuda")
            buf[:m * n] = x.view(-1)
            y = buf[shift:]
            assert bt.lib().bt_linear_forward(lin._h, None, buf.data_ptr(), m, n, code, y.data_ptr(), code, torch.cuda.current_stream().cuda_stream) == 0
            assert torch.equal(y.view(m, n), want), (m, shift)
    assert bt.lib().bt_device_check(0) == 0


def test_row_quantisers_of_tiny_rows(bt, oracle):
    # rows whose 127 / max|x| overflows, among ordinary ones, through the kernel of many rows
    n, k, m = 48, 1024, 300
    rng = np.random.default_rng(5)
    packed = ternary_packed(rng, n, k)
    x = rng.normal(0, 1, (m, k)).astype(np.float32)
    x[7] *= 1e-39
    x[250] = np.where(np.arange(k) % 3, 1e-40, -2e-40)
    lin = bt.BitLinear.from_packed(packed, [0.5], n, k)
    assert np.array_equal(lin.forward(torch.from_numpy(x).cuda()).cpu().numpy(), oracle.bitlinear_q(x, packed, [0.5], n))


@pytest.mark.parametrize("m", [1, 3, 4, 8, 9, 65, 300])  # every quantiser
@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_zeros_of_tiny_rows_stay_zeros(bt, oracle, m, dtype):
    # 127 / max|x| overflows, and a zero times infinity is no number
    n, k = 48, 1024
    rng = np.random.default_rng(6)
    packed = ternary_packed(rng, n, k)
    x = np.where(rng.random((m, k)) < 0.5, 0, rng.choice([-1, 1], (m, k)) * 2.0 ** -130).astype(np.float32)
    x = torch.from_numpy(x).to(getattr(torch, dtype))
    lin = bt.BitLinear.from_packed(packed, [0.5], n, k)
    ref = torch.from_numpy(oracle.bitlinear_q(x.float().numpy(), packed, [0.5], n)).to(x.dtype)
    assert torch.equal(lin.forward(x.cuda()).cpu(), ref)
    q, _, qsum = bt.act_quant(x.cuda())
    assert torch.equal(q.cpu() == 0, x == 0) and torch.equal(qsum.cpu(), q.cpu().sum(1, dtype=torch.int32))
    if dtype == "float32":
        assert np.array_equal(q.cpu().numpy(), oracle.act_quant(x.numpy())[0])
