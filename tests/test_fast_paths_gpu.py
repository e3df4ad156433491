"""Kernel and dispatch variants at the sizes where they can go wrong, against the dense product of the decoded weights."""

import pytest

from conftest import have_cuda, load_pkg

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
DEV = "cuda:0"


@pytest.fixture(scope="module")
def P():
    if not have_cuda():
        pytest.skip("no CUDA device")
    return load_pkg()


def _packer(P, bits):
    return {1.0: P.RootE8LatticePacker, 1.5: P.TernaryE8LatticePacker, 2.0: P.E8LatticePacker}[bits]


def _problem(P, bits, n, k, group, seed=7):
    w = P.ops.generate(n * k, seed, 0.02, torch.float16, torch.device(DEV)).view(n, k)
    packed, scales, shape = _packer(P, bits).pack(w, group)
    return packed, scales, _packer(P, bits).unpack(packed, scales, shape, torch.float32)


@pytest.mark.parametrize("bits", [1.0, 1.5, 2.0])
def test_operands_of_any_form_give_the_plain_call_s_result(P, bits):
    """Non-contiguous x, a bias of another dtype, leading dimensions: the general path equals the native call."""
    n, k, m = 96, 2048, 3
    packed, scales, wd = _problem(P, bits, n, k, 32)
    fn = {1.0: P.ops.linear_1bit, 1.5: P.ops.linear, 2.0: P.ops.linear_2bit}[bits]
    x = P.ops.generate(m * k, 8, 1.0, torch.bfloat16, torch.device(DEV)).view(m, k)
    bias = P.ops.generate(n, 9, 0.5, torch.bfloat16, torch.device(DEV))
    plain = fn(x, packed, scales, bias, n, k, 32)
    ref = x.float() @ wd.t() + bias.float()
    assert float((plain.float() - ref).norm() / ref.norm()) <= 4e-3
    assert torch.equal(plain, fn(x.t().contiguous().t(), packed, scales, bias.float(), n, k, 32))
    layer = P.E8LatticeLinear(k, n, bias=True, group_size=32, bitrate=bits, device=DEV, dtype=torch.bfloat16)
    layer.packed_weight.copy_(packed)
    layer.block_scales.copy_(scales)
    with torch.no_grad():
        layer.bias.copy_(bias)
        assert torch.equal(layer(x.view(m, 1, k)), plain.view(m, 1, n))          # native call
    y = layer(x.clone().requires_grad_(True))                                    # autograd node
    assert y.requires_grad and torch.equal(y.detach(), plain)


@pytest.mark.parametrize("bits,group", [(1.5, 32), (1.5, 16), (2.0, 32), (2.0, 8), (1.0, 32), (1.0, 16), (1.0, 8)])
@pytest.mark.parametrize("m,n,k", [(17, 40, 32), (130, 72, 288), (333, 520, 736), (64, 129, 2080)])
def test_batches_of_tokens_with_k_a_multiple_of_32(P, bits, group, m, n, k):
    """K that is no multiple of 256: rows start at any even address and the last 256-wide chunk is cut short."""
    packed, scales, wd = _problem(P, bits, n, k, group)
    fn = {1.0: P.ops.linear_1bit, 1.5: P.ops.linear, 2.0: P.ops.linear_2bit}[bits]
    fmt, gemm = {1.0: 1, 1.5: 0, 2.0: 2}[bits], P._cabi.OJX_LINEAR_GEMM
    for dt in (torch.bfloat16, torch.float16):
        x = P.ops.generate(m * k, 8, 1.0, dt, torch.device(DEV)).view(m, k)
        ref, bound = x.double() @ wd.double().t(), x.double().abs() @ wd.double().abs().t()     # unrounded weights: of every format exact here
        for flags, limit in ((gemm, 2e-5), (0, 5e-6)):                   # fp32 outputs: the tcgen05 kernel, and the decode kernel that serves them
            y = P.ops._linear(fmt, x, packed, scales, None, n, k, group, torch.float32, flags)
            assert float(((y.double() - ref).abs() / (bound + 1e-20)).max()) <= limit
        assert torch.equal(fn(x, packed, scales, None, n, k, group), P.ops._linear(fmt, x, packed, scales, None, n, k, group, None, gemm))
    P.ops.gemm_status(torch.device(DEV))


@pytest.mark.parametrize("group", [8, 32, 64])
def test_root_packer_on_ties_zeros_and_non_finite_values(P, oracle, group):
    """The pruned search against the oracle's walk over all 256 vectors where magnitudes coincide, vanish or are not finite."""
    g = torch.Generator().manual_seed(3)
    w = torch.randn(64, 512, generator=g)
    w[8:16] = torch.round(w[8:16] * 2) / 2                              # many equal magnitudes
    w[16:24] *= (torch.rand(8, 512, generator=g) < 0.4)                 # most magnitudes zero
    w[24:32] = w[24:32].sign() * 0.37                                   # all equal
    w[32:40] *= torch.where(torch.rand(8, 512, generator=g) < 0.3, 1e-7, 1.0)
    w[40, ::64] = 0.0
    w[41] = 0.0
    for dt in (torch.float32, torch.bfloat16, torch.float16):
        wt = w.to(dt)
        packed, scales, _ = P.RootE8LatticePacker.pack(wt.to(DEV), group)
        p_ref, s_ref, _ = oracle.encode_1bit(wt.float().numpy(), group)
        assert (packed.cpu().numpy() == p_ref).all()
        assert (scales.view(torch.int16).cpu().numpy().view("uint16") == s_ref.view("uint16")).all()


_DECODE_SHAPES = [(1, 256), (17, 512), (100, 4096), (1000, 4352), (65, 14336), (2500, 8448), (33, 32), (40, 96), (129, 2912), (50, 11040)]


@pytest.mark.parametrize("bits,group", [(1.5, 32), (1.5, 16), (2.0, 32), (2.0, 16), (2.0, 8), (1.0, 32), (1.0, 16), (1.0, 8)])
@pytest.mark.parametrize("n,k", _DECODE_SHAPES)
def test_decode_kernels_at_the_edges_of_their_tiles(P, bits, group, n, k):
    """One row of weights, remainders of a tile, one and several chunks of K (clusters that split them), K of any number of 32s."""
    packed, scales, wd = _problem(P, bits, n, k, group)             # fp32: the weights as they are, whatever the batch
    fmt = {1.0: 1, 1.5: 0, 2.0: 2}[bits]
    for m in (1, 2, 3, 8, 9, 16):
        for dt in (torch.bfloat16, torch.float16):
            x = P.ops.generate(m * k, 8 + m, 1.0, dt, torch.device(DEV)).view(m, k).clone()
            x[:, ::97] *= 30
            bias = P.ops.generate(n, 9, 0.5, dt, torch.device(DEV))
            y = P.ops._linear(fmt, x, packed, scales, bias, n, k, group, torch.float32, P._cabi.OJX_LINEAR_DECODE)
            ref = x.double() @ wd.double().t() + bias.double()
            bound = x.double().abs() @ wd.double().abs().t() + bias.double().abs()
            assert float(((y.double() - ref).abs() / bound.clamp_min(1e-30)).max()) <= 5e-6, (m, dt)


@pytest.mark.parametrize("bits,group,k", [(2.0, 8, 4096), (2.0, 32, 14336), (1.5, 16, 8192), (1.0, 8, 2080)])
def test_decode_kernels_keep_non_finite_activations_in_their_row(P, bits, group, k):
    n, m = 48, 5
    packed, scales, wd = _problem(P, bits, n, k, group)
    fmt = {1.0: 1, 1.5: 0, 2.0: 2}[bits]
    x = P.ops.generate(m * k, 3, 1.0, torch.bfloat16, torch.device(DEV)).view(m, k).clone()
    x[1] *= 2.0 ** 20
    x[4] *= 2.0 ** 112
    x[1, k - 5] = float("inf")
    x[3, 7] = float("nan")
    y = P.ops._linear(fmt, x, packed, scales, None, n, k, group, torch.float32, P._cabi.OJX_LINEAR_DECODE)
    ref = x.float() @ wd.t()
    assert torch.equal(torch.isnan(y), torch.isnan(ref)) and torch.equal(torch.isinf(y), torch.isinf(ref))
    for row in (0, 2, 4):
        assert float((y[row].double() - ref[row].double()).norm() / ref[row].double().norm()) < 1e-3


@pytest.mark.parametrize("m", [1, 4, 12])
def test_grouped_launch_over_many_matrices_of_different_shapes(P, m):
    """Work items that run across matrix borders, tables of more entries than a CTA has threads' worth of items, K of one and of
    several chunks in one launch."""
    dev = torch.device(DEV)
    for count in (2, 40, 300):
        entries, shapes, want = [], [], []
        for i in range(count):
            n, k = (48, 256) if count == 300 else (16 * (1 + i % 5) + (i % 3), 256 * (1 + (7 * i) % 19))
            packed, scales, _ = _problem(P, 1.5, n, k, 32, seed=i)
            x = P.ops.generate(m * k, 50 + i, 1.0, torch.bfloat16, dev).view(m, k)
            y = torch.empty((m, n), dtype=torch.bfloat16, device=dev)
            entries.append((x, packed, scales, None, y))
            shapes.append((n, k))
            want.append(P.ops.linear(x, packed, scales, None, n, k, 32))
        P.ops.GroupedGemv(entries, shapes)()
        for e, w in zip(entries, want):
            assert float((e[4].float() - w.float()).norm() / w.float().norm()) <= 4e-3


@pytest.mark.parametrize("bits,group,n,k,rank,had", [(1.5, 32, 72, 4096, 16, True), (1.5, 16, 33, 96, 3, True), (2.0, 8, 40, 2912, 8, False),
                                                     (2.0, 32, 64, 2048, 64, True), (1.0, 32, 48, 8192, 17, False), (1.0, 16, 100, 320, 1, True)])
def test_adapter_layer_at_decode_shapes_in_one_call(P, bits, group, n, k, rank, had):
    """Ranks that fill a slab of sixteen columns, less and more; K of less than one group per CTA; every row count of a block."""
    dev = torch.device(DEV)
    for dt in (torch.bfloat16, torch.float16):
        lin = torch.nn.Linear(k, n, bias=True).to(dev).to(dt)
        layer = P.E8LatticeLinear.from_linear(lin, rank=rank, bitrate=bits, group_size=group, use_hadamard=had).requires_grad_(False)
        layer.lora_B.copy_(torch.randn_like(layer.lora_B) * 0.1)
        wd = layer.unpack_weights(torch.float32).double()
        for m in (1, 2, 4, 5, 8, 9, 16):
            x = P.ops.generate(m * k, 8 + m, 1.0, dt, dev).view(1, m, k)
            y = P.ops.layer_forward_adapter({1.0: 1, 1.5: 0, 2.0: 2}[bits], x, layer.packed_weight, layer.block_scales, layer.bias, n, k, group,
                                            had, layer.lora_A, layer.lora_B, layer.scaling, torch.float32)
            assert y is not None and y.shape == (1, m, n)
            low = layer.scaling * ((x.double() @ layer.lora_A.double()) @ layer.lora_B.double())
            ref = x.double() @ wd.t() + layer.bias.double() + low
            assert float((y.double() - ref).norm() / ref.norm()) < (5e-3 if had and dt == torch.bfloat16 else 1.5e-3), (dt, m)
            assert float((layer(x).double() - ref).norm() / ref.norm()) < 8e-3, (dt, m)


def test_adapter_layer_on_a_batch_of_tokens(P):
    dev = torch.device(DEV)
    lin = torch.nn.Linear(512, 264, bias=True).to(dev).to(torch.bfloat16)
    layer = P.E8LatticeLinear.from_linear(lin, rank=8, bitrate=1.5, group_size=32)
    with torch.no_grad():
        layer.lora_B.copy_(torch.randn_like(layer.lora_B) * 0.1)
    x = torch.randn(2, 20, 512, device=dev).to(torch.bfloat16)
    ref = (x.double() @ layer.unpack_weights(torch.float32).double().t() + layer.bias.double()
           + layer.scaling * ((x.double() @ layer.lora_A.double()) @ layer.lora_B.double()))
    with torch.no_grad():
        y = layer(x)
    y_grad = layer(x)
    assert y.shape == y_grad.shape == (2, 20, 264) and y_grad.requires_grad
    for v in (y, y_grad):
        assert float((v.double() - ref).norm() / ref.norm()) < 8e-3


@pytest.mark.parametrize("rows,cols,group", [(1, 3, 8), (5, 1023, 8), (7, 4096, 32), (33, 1021, 24), (1025, 33, 16)])
def test_unpack_2bit_at_the_edges_of_its_chunks(P, rows, cols, group):
    """Fewer weights than a chunk, a last chunk that is cut short, groups that are no power of two: every type against the fp32 values."""
    dev = torch.device(DEV)
    packed, scales = P.ops.encode_2bit(P.ops.generate(rows * cols, 5, 1.0, torch.float32, dev).view(rows, cols), group)
    codes = torch.stack([(packed.int() >> (2 * i)) & 3 for i in range(4)], 1).reshape(-1)[:rows * cols]
    index = torch.arange(rows * cols, device=dev) // group
    for dt in (torch.float32, torch.float16, torch.bfloat16):
        got = P.ops.decode_2bit(packed, scales, (rows, cols), dt)
        want = (codes.float() - 1.5) * scales[index].to(dt).float()
        assert torch.equal(got, want.to(dt).view(rows, cols)), dt


@pytest.mark.parametrize("rows,cols,group", [(1, 3, 8), (5, 1023, 8), (33, 1021, 24)])
def test_unpack_1bit_at_the_edges_of_its_codes(P, rows, cols, group):
    """A last code that is cut short, groups that are no power of two; every type against the fp32 values of whole codes."""
    dev = torch.device(DEV)
    total, codes = rows * cols, (rows * cols + 7) // 8
    packed, scales = P.ops.encode_1bit(P.ops.generate(total, 5, 1.0, torch.float32, dev).view(rows, cols), group)
    unit = P.ops.decode_1bit(packed, torch.ones(-(-codes * 8 // group), dtype=torch.float16, device=dev), (codes, 8), torch.float32)
    index = torch.arange(total, device=dev) // group
    for dt in (torch.float32, torch.float16, torch.bfloat16):
        want = unit.reshape(-1)[:total] * scales[index].to(dt).float()
        assert torch.equal(P.ops.decode_1bit(packed, scales, (rows, cols), dt), want.to(dt).view(rows, cols)), dt


@pytest.mark.parametrize("bits,group,k", [(1.5, 32, 512), (1.5, 16, 288), (2.0, 8, 512), (2.0, 32, 96), (1.0, 32, 512), (1.0, 8, 96)])
def test_buffers_too_short_for_the_shape_are_refused(P, bits, group, k):
    """Codes or scales of one row fewer: every entry point raises before anything is launched; longer buffers are taken."""
    n, dev = 48, torch.device(DEV)
    packed, scales, _ = _problem(P, bits, n, k, group)
    fmt = {1.0: 1, 1.5: 0, 2.0: 2}[bits]
    fn = {1.0: P.ops.linear_1bit, 1.5: P.ops.linear, 2.0: P.ops.linear_2bit}[bits]
    short = [(packed[:-packed.numel() // n], scales), (packed, scales[:-1])]
    lora_a, lora_b = torch.zeros(k, 8, dtype=torch.bfloat16, device=dev), torch.zeros(8, n, dtype=torch.bfloat16, device=dev)
    for m in (1, 8, 40):
        x, gy = torch.randn(m, k, device=dev).bfloat16(), torch.randn(m, n, device=dev).bfloat16()
        y = fn(x, packed, scales, None, n, k, group)
        assert torch.equal(y, fn(x, torch.cat([packed, packed]), torch.cat([scales, scales]), None, n, k, group))
        for pk, sc in short:
            with pytest.raises(ValueError):
                fn(x, pk, sc, None, n, k, group)
            with pytest.raises(ValueError):
                fn(x.float(), pk, sc, None, n, k, group)
            with pytest.raises(ValueError):
                P.ops.linear_dx(gy, pk, sc, n, k, group) if fmt == 0 else P.ops.linear_dx_lowbit(fmt, gy, pk, sc, n, k, group)
            assert P.ops.layer_forward(fmt, x, pk, sc, None, n, k, group, False) is None
            assert P.ops.layer_forward_adapter(fmt, x, pk, sc, None, n, k, group, False, lora_a, lora_b, 1.0) is None
            layer = P.E8LatticeLinear(k, n, bias=False, rank=8, group_size=group, bitrate=bits, device=dev, dtype=torch.bfloat16)
            layer.packed_weight, layer.block_scales = pk, sc
            with torch.no_grad(), pytest.raises(ValueError):
                layer(x)


@pytest.mark.parametrize("bits", [1.0, 2.0])
def test_sibling_unpackers_refuse_buffers_too_short_for_the_shape(P, bits):
    packed, scales, _ = _problem(P, bits, 64, 2048, 32)
    with pytest.raises(ValueError):
        P.ops._decode_lowbit(int(bits), packed, scales, (65, 2048), torch.float32)


@pytest.mark.parametrize("bits", [1.0, 2.0])
def test_sibling_formats_on_buffers_with_strides(P, bits):
    """Codes and scales that are every other element of a wider buffer give what contiguous ones give."""
    n, k, m, fmt, dev = 64, 2048, 3, int(bits), torch.device(DEV)
    packed, scales, _ = _problem(P, bits, n, k, 32)
    wide_pk, wide_sc = torch.stack([packed, ~packed], 1)[:, 0], torch.stack([scales, scales + 1], 1)[:, 0]
    gy, t = torch.randn(m, n, device=dev).bfloat16(), torch.randn(m, 8, device=dev)
    x, b = torch.randn(m, k, device=dev).bfloat16(), torch.randn(8, n, device=dev).bfloat16()
    for fn in (lambda p, s: P.ops.linear_dx_lowbit(fmt, gy, p, s, n, k, 32), lambda p, s: P.ops._decode_lowbit(fmt, p, s, (n, k), torch.float32),
               lambda p, s: P.ops.linear_lowbit_lora(fmt, x, p, s, None, n, k, 32, t, b)):
        assert torch.equal(fn(packed, scales), fn(wide_pk, wide_sc))


@pytest.mark.parametrize("bits,group,n,k", [(2.0, 32, 50, 4096), (2.0, 8, 17, 512), (2.0, 16, 40, 2912), (2.0, 32, 33, 14336),
                                            (1.0, 32, 50, 4096), (1.0, 8, 17, 512), (1.0, 16, 40, 2912), (1.0, 32, 33, 14336)])
def test_decode_kernels_with_scales_near_the_top_of_fp16(P, bits, group, n, k):
    """Twice a scale above 32752 is no fp16 number: such rows still give the fp32 product, alone and with an adapter's term."""
    packed, scales, _ = _problem(P, bits, n, k, group)
    fmt, dev = int(bits), torch.device(DEV)
    scales = scales.clone()
    scales.view(n, -1)[3::4, ::5] = 33000.0
    scales.view(n, -1)[7, 1] = 65504.0
    wd = _packer(P, bits).unpack(packed, scales, (n, k), torch.float32).double()
    a, b = torch.randn(k, 4, device=dev), torch.randn(4, n, device=dev)
    for m in (1, 2, 5, 9, 16):
        for dt in (torch.bfloat16, torch.float16):
            x = P.ops.generate(m * k, 8 + m, 1.0, dt, dev).view(m, k)
            y = P.ops._linear(fmt, x, packed, scales, None, n, k, group, torch.float32, P._cabi.OJX_LINEAR_DECODE)
            ref, bound = x.double() @ wd.t(), x.double().abs() @ wd.abs().t()
            assert float(((y.double() - ref).abs() / bound.clamp_min(1e-30)).max()) <= 5e-6, (m, dt)
            y = P.ops.layer_forward_adapter(fmt, x, packed, scales, None, n, k, group, False, a.to(dt), b.to(dt), 0.5, torch.float32)
            low = 0.5 * ((x.double() @ a.to(dt).double()) @ b.to(dt).double())
            bound += 0.5 * ((x.double().abs() @ a.to(dt).double().abs()) @ b.to(dt).double().abs())
            assert float(((y.double() - ref - low).abs() / bound.clamp_min(1e-30)).max()) <= 5e-6, (m, dt)


@pytest.mark.parametrize("bits", [2.0, 1.0])
@pytest.mark.parametrize("group,m,n,k", [(32, 40, 136, 2912), (8, 130, 40, 544), (16, 17, 33, 96), (32, 300, 300, 4128)])
def test_batches_of_tokens_over_scales_of_every_size(P, bits, group, m, n, k):
    """K that is no multiple of 256: scales whose 1.5- or 2-fold fp16 does not have, and ones whose halves it does not, in rows of
    their own and beside ordinary ones; Inf and NaN stay in their token and give the dense product's pattern."""
    packed, scales, _ = _problem(P, bits, n, k, group)
    call = lambda x: P.ops._linear(int(bits), x, packed, scales, None, n, k, group, torch.float32, P._cabi.OJX_LINEAR_GEMM)
    scales = scales.clone()
    rows = scales.view(n, -1)
    rows[1::8, ::2] = 65504.0
    rows[2::8] = 44000.0
    rows[3::8] *= 2.0 ** -14
    rows[4::8] = 2.0 ** -24 * torch.randint(1, 4, rows[4::8].shape, device=DEV)
    rows[5::8] = 0.0
    wd = _packer(P, bits).unpack(packed, scales, (n, k), torch.float32).double()
    for dt in (torch.bfloat16, torch.float16):
        x = P.ops.generate(m * k, 8, 1.0, dt, torch.device(DEV)).view(m, k).clone()
        y = call(x)
        ref, bound = x.double() @ wd.t(), x.double().abs() @ wd.abs().t()
        assert float(((y.double() - ref).abs() / bound.clamp_min(1e-35)).max()) <= 2e-5, dt
        x[3, k - 1], x[9, 5], x[10, 0] = float("inf"), float("nan"), -float("inf")
        y2, ref = call(x), x.float() @ wd.float().t()
        assert torch.equal(torch.isnan(y2), torch.isnan(ref)) and torch.equal(torch.isinf(y2), torch.isinf(ref))
        keep = [i for i in range(m) if i not in (3, 9, 10)]
        assert torch.equal(y2[keep], y[keep])
    P.ops.gemm_status(torch.device(DEV))


@pytest.mark.parametrize("bits,group", [(1.5, 32), (1.5, 16), (2.0, 8), (1.0, 32)])
@pytest.mark.parametrize("m,n,k", [(1, 40, 256), (3, 33, 4096), (20, 24, 288)])
def test_activations_that_are_not_aligned_take_the_fp32_kernels(P, bits, group, m, n, k):
    """x at an address that is no multiple of 16: the scalar kernel of the format, 16-bit and fp32 activations."""
    packed, scales, wd = _problem(P, bits, n, k, group)
    fn = {1.0: P.ops.linear_1bit, 1.5: P.ops.linear, 2.0: P.ops.linear_2bit}[bits]
    for dt in (torch.bfloat16, torch.float16, torch.float32):
        x = P.ops.generate(m * k + 1, 8, 1.0, dt, torch.device(DEV))[1:].view(m, k)
        y = fn(x, packed, scales, None, n, k, group, out_dtype=torch.float32)
        ref, bound = x.double() @ wd.double().t(), x.double().abs() @ wd.double().abs().t()
        assert float(((y.double() - ref).abs() / bound.clamp_min(1e-30)).max()) <= 2e-6, dt


@pytest.mark.parametrize("bits", [1.5, 2.0, 1.0])
@pytest.mark.parametrize("n,k", [(40, 512), (40, 288), (24, 8224)])
def test_batches_of_tokens_with_large_values_beside_infinities(P, bits, n, k):
    """A token with an infinity and finite values that fp16 does not have: they stay finite, so that the dense product's Inf is no NaN."""
    m = 20
    packed, scales, wd = _problem(P, bits, n, k, 32)
    fn = {1.0: P.ops.linear_1bit, 1.5: P.ops.linear, 2.0: P.ops.linear_2bit}[bits]
    x = P.ops.generate(m * k, 8, 1.0, torch.bfloat16, torch.device(DEV)).view(m, k).clone()
    x[:, 1::7] *= 1e20
    x[3, 5], x[7, k - 1], x[9, 0] = float("inf"), -float("inf"), float("nan")
    y, ref = fn(x, packed, scales, None, n, k, 32), x.float() @ wd.t()
    assert torch.equal(torch.isnan(y), torch.isnan(ref)) and torch.equal(torch.isinf(y), torch.isinf(ref))
    keep = [i for i in range(m) if i not in (3, 7, 9)]
    assert float((y[keep].double() - ref[keep].double()).norm() / ref[keep].double().norm()) <= 4e-3
