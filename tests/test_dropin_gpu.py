"""GPU tests of the drop-in surface beyond single kernels: the Walsh-Hadamard option end to end against
vectors produced by the reference, model packing, streaming row blocks into a layer, the full-size
benchmark shapes at the batch sizes the other files leave out, and - where the reference package can be
imported - the reference's own layer running on CUDA through the patched kernel seam."""

import math
import os
import sys

import numpy as np
import pytest

from conftest import ROOT, have_cuda, load_pkg

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

DEV = "cuda:0"


@pytest.fixture(scope="module")
def P():
    if not have_cuda():
        pytest.skip("no CUDA device")
    pkg = load_pkg()
    pkg._cabi.lib()
    return pkg


def f16_bits(t):
    return t.view(torch.int16).cpu().numpy().view(np.uint16)


def test_fwht_matches_reference_bits_on_device(P, golden):
    _, arrays = golden
    for tag, dt in (("f32", torch.float32), ("f16", torch.float16), ("bf16", torch.bfloat16)):
        x = torch.from_numpy(arrays[f"fwht/{tag}/input"]).to(dt).to(DEV)
        y = P.fwht_block32(x).float().cpu().numpy()
        ref = arrays[f"fwht/{tag}/output"]
        if tag == "f32":
            # CUDA and CPU both evaluate the same additions in the same order: identical bits
            assert np.array_equal(y.view(np.uint32), ref.view(np.uint32))
        else:
            assert np.array_equal(y, ref)


def test_hadamard_layer_matches_reference(P, golden, oracle):
    """A layer packed and run with use_hadamard=True: packed bytes and scales equal the reference's bit for
    bit, unpack_weights equals its rotated weights, and the forward (fp32 activations, so nothing but the
    summation order differs) matches its output (ojasx2/math/lattice.py:564-567,807,825)."""
    meta, arrays = golden
    h = meta["hadamard"]
    k, n, b = h["in_features"], h["out_features"], h["batch"]
    lin = torch.nn.Linear(k, n, bias=True)
    with torch.no_grad():
        lin.weight.copy_(torch.from_numpy(oracle.gen_normal(h["weight_seed"], n * k, 0.02).reshape(n, k).copy()))
        lin.bias.copy_(torch.from_numpy(oracle.gen_normal(h["bias_seed"], n, 0.1).copy()))
    layer = P.E8LatticeLinear.from_linear(lin.to(DEV), bitrate=1.5, group_size=32, use_hadamard=True)
    assert layer.use_hadamard
    assert np.array_equal(layer.packed_weight.cpu().numpy(), arrays["hadamard/packed"])
    assert np.array_equal(f16_bits(layer.block_scales), arrays["hadamard/scales"])
    w = layer.unpack_weights(torch.float32).detach().cpu().numpy()
    assert np.allclose(w, arrays["hadamard/unpacked"], rtol=0, atol=1e-7)
    x = torch.from_numpy(oracle.gen_normal(h["x_seed"], b * k, 1.0).reshape(b, k).copy()).to(DEV)
    y = layer(x).detach().cpu().numpy()
    ref = arrays["hadamard/y"]
    assert np.linalg.norm(y - ref) <= 1e-5 * np.linalg.norm(ref)
    # bf16 activations through the tensor-core decode kernel stay inside the GEMM contract
    yb = layer(x.bfloat16()).detach().float().cpu().numpy()
    # (the rotation itself then runs in bf16, as in the reference, which rotates x in its own dtype)
    assert np.linalg.norm(yb - ref) <= 2e-2 * np.linalg.norm(ref)


def test_pack_model_e8_replaces_and_runs(P):
    dev = torch.device(DEV)
    torch.manual_seed(0)

    class Block(torch.nn.Module):
        def __init__(self):
            super().__init__()
            self.q_proj = torch.nn.Linear(256, 256, bias=False)
            self.up_proj = torch.nn.Linear(256, 512, bias=True)
            self.lm_head = torch.nn.Linear(512, 64, bias=False)
            self.norm = torch.nn.LayerNorm(256)

        def forward(self, x):
            return self.lm_head(torch.relu(self.up_proj(self.q_proj(self.norm(x)))))

    model = torch.nn.Sequential(Block()).to(dev)
    x = torch.randn(3, 256, device=dev)
    packed = P.pack_model_e8(model, rank=2, group_size=32, bitrate=1.5, exclude_modules=["lm_head"], inplace=False)
    blk, orig = packed[0], model[0]
    assert isinstance(blk.q_proj, P.E8LatticeLinear) and isinstance(blk.up_proj, P.E8LatticeLinear)
    assert isinstance(blk.lm_head, torch.nn.Linear) and isinstance(orig.q_proj, torch.nn.Linear)   # excluded / not in place
    assert blk.q_proj.rank == 2 and blk.q_proj.bias is None and blk.up_proj.bias is not None
    # each packed layer computes x . dequant(W)^T + bias with exactly the weights it reports
    h = blk.norm(x)
    ref = torch.nn.functional.linear(h, blk.q_proj.unpack_weights(torch.float32))
    assert float((blk.q_proj(h) - ref).norm() / ref.norm()) < 1e-5
    y = packed(x)
    assert tuple(y.shape) == (3, 64) and torch.isfinite(y).all()
    only_q = P.pack_model_e8(model, bitrate=1.5, target_modules="q_proj", inplace=False)
    assert isinstance(only_q[0].q_proj, P.E8LatticeLinear) and isinstance(only_q[0].up_proj, torch.nn.Linear)


def test_copy_row_block_into_layer_streams_a_matrix(P, oracle):
    """Row blocks fed one at a time (the safetensors streaming path, ojasx2/streaming_e8.py:162-193) fill the
    layer's buffers with the same bytes as packing the whole matrix."""
    dev = torch.device(DEV)
    st = __import__("importlib").import_module(P.__name__ + ".streaming_e8")
    n, k = 70, 512
    w = torch.from_numpy(oracle.gen_normal(91, n * k, 0.02).reshape(n, k).copy())
    for had in (False, True):
        layer = P.E8LatticeLinear(k, n, bias=False, group_size=32, bitrate=1.5, use_hadamard=had, device=dev)
        consumed = 0
        for r0 in range(0, n, 16):
            consumed += st._copy_row_block_into_layer(layer, r0, w[r0: r0 + 16].half(), had)      # host fp16 blocks
        assert consumed == n * k * 2
        src = P.fwht_block32(w.half().to(dev)) if had else w.half().to(dev)
        pk, sc, _ = P.TernaryE8LatticePacker.pack(src, 32)
        assert torch.equal(layer.packed_weight, pk) and torch.equal(layer.block_scales, sc)
    with pytest.raises(ValueError):
        st._copy_row_block_into_layer(layer, 0, w[:4, :100], False)
    with pytest.raises(TypeError):
        st._copy_row_block_into_layer(layer, 0, torch.zeros(4, k, dtype=torch.int32), False)
    with pytest.raises(RuntimeError):
        st._copy_row_block_into_layer(layer, n - 2, w[:4], False)


SHAPES_KN = [(4096, 4096), (4096, 1024), (4096, 14336), (14336, 4096)]


def _check_against_dense(P, k, n, m, force):
    dev = torch.device(DEV)
    w = P.ops.generate(n * k, 31 + n + k, 0.02, torch.float16, dev).view(n, k)
    pk, sc = P.ops.encode(w, 32)
    del w
    wd = P.ops.decode(pk, sc, (n, k), torch.float32)                       # bit-exact against the oracle elsewhere
    x = P.ops.generate(m * k, 5 + m, 1.0, torch.bfloat16, dev).view(m, k)
    bias = P.ops.generate(n, 6 + m, 0.1, torch.bfloat16, dev)
    y = P.ops.linear(x, pk, sc, bias, n, k, 32, force=force)
    if force == "gemm":
        P.ops.gemm_status(dev)
    ref = x.float() @ wd.t() + bias.float()
    d = y.float() - ref
    assert float(d.norm() / ref.norm()) <= 2e-3, (k, n, m)
    assert float(d.abs().max()) <= 1e-2 * float(x.float().abs().max()) * math.sqrt(k), (k, n, m)


@pytest.mark.parametrize("k,n", SHAPES_KN)
def test_decode_batch4_full_size_shapes(P, k, n):
    _check_against_dense(P, k, n, 4, "gemv")


@pytest.mark.parametrize("k,n", SHAPES_KN[1:])
def test_prefill_2048_tokens_full_size_shapes(P, k, n):
    """4096 -> 1024 (fewer tiles than SMs), 4096 -> 14336 (three waves plus a tail launch) and
    14336 -> 4096 (long rows: the two-pass activation normalisation); 4096 -> 4096 is covered elsewhere."""
    _check_against_dense(P, k, n, 2048, "gemm")


@pytest.mark.parametrize("k,n,m,dt", [(256, 64, 16, torch.float16), (512, 200, 300, torch.bfloat16), (4096, 1024, 2048, torch.bfloat16),
                                       (1024, 4096, 513, torch.bfloat16), (14336, 4096, 256, torch.float16)])
def test_backward_dx_kernel_matches_dense_product(P, k, n, m, dt):
    """dX = dY . W from the packed codes (contraction over the weight rows on the tensor cores) against a dense fp32
    product with the bit-exact decoded weights: ragged token blocks, a contraction length that is not a multiple
    of the 64-row block, long and short contractions."""
    dev = torch.device(DEV)
    w = P.ops.generate(n * k, 700 + n, 0.02, torch.float16, dev).view(n, k)
    pk, sc = P.ops.encode(w, 32)
    del w
    wd = P.ops.decode(pk, sc, (n, k), torch.float32)
    gy = P.ops.generate(m * n, 701 + m, 1.0, dt, dev).view(m, n)
    gy[1] *= 1.0e3
    gy[m - 1] *= 1.0e-3
    dx = P.ops.linear_dx(gy, pk, sc, n, k, 32)
    P.ops.gemm_status(dev)
    assert dx.dtype == dt and tuple(dx.shape) == (m, k)
    ref = gy.float() @ wd
    for rows in (slice(0, 1), slice(1, 2), slice(m - 1, m), slice(0, m)):
        d = dx[rows].float() - ref[rows]
        assert float(d.norm() / ref[rows].norm()) <= 2e-3, (k, n, m, rows)
    dx32 = P.ops.linear_dx(gy, pk, sc, n, k, 32, out_dtype=torch.float32)
    assert float((dx32 - ref).norm() / ref.norm()) <= 2e-5            # fp32 accumulation of exact products


def test_autograd_backward_uses_the_packed_weights(P):
    dev = torch.device(DEV)
    lin = torch.nn.Linear(512, 96, bias=True).to(dev)
    layer = P.E8LatticeLinear.from_linear(lin, bitrate=1.5, group_size=32)
    x = torch.randn(6, 7, 512, device=dev, dtype=torch.bfloat16, requires_grad=True)
    y = layer(x)
    gy = torch.randn_like(y)
    y.backward(gy)
    w = layer.unpack_weights(torch.float32)
    ref = gy.float().reshape(-1, 96) @ w
    assert x.grad.dtype == torch.bfloat16
    assert float((x.grad.float().reshape(-1, 512) - ref).norm() / ref.norm()) <= 4e-3        # bf16 output rounding
    assert layer.bias.grad is not None and float((layer.bias.grad.float() - gy.float().sum((0, 1))).abs().max()) < 0.1


def test_registered_operators_and_compile_without_graph_breaks(P):
    """torch.ops.ojasx_math_native.fused_ternary_e8_gemm_fwd / _bwd_dx with the reference's schema strings
    (ojasx_math_bindings.cpp:592-595): callable on CUDA tensors, shape-inferable on meta tensors, and a packed layer
    with LoRA compiles as ONE graph (fullgraph=True) and gives the eager result, forward and backward."""
    dev = torch.device(DEV)
    ns = torch.ops.ojasx_math_native
    fwd = ns.fused_ternary_e8_gemm_fwd.default
    assert str(fwd._schema) == ("ojasx_math_native::fused_ternary_e8_gemm_fwd(Tensor x, Tensor packed_weight, Tensor block_scales, "
                                "Tensor? bias=None, int group_size=32) -> Tensor")
    assert str(ns.fused_ternary_e8_gemm_bwd_dx.default._schema) == (
        "ojasx_math_native::fused_ternary_e8_gemm_bwd_dx(Tensor grad_y, Tensor packed_weight, Tensor block_scales, "
        "int in_features, int group_size=32) -> Tensor")
    n, k, m = 192, 512, 6
    lin = torch.nn.Linear(k, n, bias=True).to(dev)
    layer = P.E8LatticeLinear.from_linear(lin, rank=4, bitrate=1.5, group_size=32)
    with torch.no_grad():
        layer.lora_B.normal_(0, 0.02)
    pk2, sc2 = layer.packed_weight.view(n, -1), layer.block_scales.view(n, -1)
    x = torch.randn(m, k, device=dev, dtype=torch.bfloat16)
    y_op = ns.fused_ternary_e8_gemm_fwd(x, pk2, sc2, layer.bias.detach().bfloat16(), 32)
    assert torch.equal(y_op, P.ops.linear(x, layer.packed_weight, layer.block_scales, layer.bias.detach(), n, k, 32))
    meta = ns.fused_ternary_e8_gemm_fwd(x.to("meta"), pk2.to("meta"), sc2.to("meta"), None, 32)
    assert meta.device.type == "meta" and tuple(meta.shape) == (m, n) and meta.dtype == torch.bfloat16
    gmeta = ns.fused_ternary_e8_gemm_bwd_dx(y_op.to("meta"), pk2.to("meta"), sc2.to("meta"), k, 32)
    assert tuple(gmeta.shape) == (m, k)

    compiled = torch.compile(layer, fullgraph=True, backend="aot_eager")
    xe = x.clone().requires_grad_(True)
    xc = x.clone().requires_grad_(True)
    ye = layer(xe)
    yc = compiled(xc)
    assert torch.equal(ye, yc)
    g = torch.randn_like(ye)
    ye.backward(g)
    ge_b = layer.lora_B.grad.clone()
    layer.zero_grad()
    yc.backward(g)
    assert torch.allclose(xe.grad.float(), xc.grad.float(), rtol=2e-2, atol=2e-2)
    assert torch.allclose(ge_b.float(), layer.lora_B.grad.float(), rtol=2e-2, atol=2e-2)


def test_activation_outliers_nan_and_inf(P, oracle):
    """One huge activation per 256-wide slice must not wipe out its neighbours, and non-finite activations
    must show up in the outputs the way a dense product shows them (rows of the batch they belong to)."""
    dev = torch.device(DEV)
    n, k = 96, 4096
    w = P.ops.generate(n * k, 17, 0.02, torch.float16, dev).view(n, k)
    pk, sc = P.ops.encode(w, 32)
    wd = P.ops.decode(pk, sc, (n, k), torch.float32)
    for m in (1, 4, 16):
        x = P.ops.generate(m * k, 18 + m, 1.0, torch.bfloat16, dev).view(m, k).clone()
        for mag in (1.0e2, 1.0e4):
            xo = x.clone()
            xo[:, 7::256] *= mag                                               # one outlier in every slice of every row
            y = P.ops.linear(xo, pk, sc, None, n, k, 32, out_dtype=torch.float32)
            # per-output bound relative to sum |x_k| |w_k| of that output (what fp32 accumulation of exact
            # products can be held to), not to the outlier
            ref = xo.float() @ wd.t()
            magnitude = xo.float().abs() @ wd.abs().t()
            assert float(((y - ref).abs() / magnitude).max()) < 1e-5, (m, mag)
        xn = x.clone()
        xn[0, 100] = float("nan")
        y = P.ops.linear(xn, pk, sc, None, n, k, 32, out_dtype=torch.float32)
        assert torch.isnan(y[0]).all()
        if m > 1:
            assert torch.isfinite(y[1:]).all()
        xi = x.clone()
        xi[m - 1, 3000] = float("inf")
        y = P.ops.linear(xi, pk, sc, None, n, k, 32, out_dtype=torch.float32)
        assert (~torch.isfinite(y[m - 1])).all()
        if m > 1:
            assert torch.isfinite(y[: m - 1]).all()
        # the pattern of NaN / +Inf / -Inf equals that of the dense fp32 product (0 * Inf = NaN, w * Inf = +-Inf)
        xi[m - 1, 17] = float("-inf")
        xi[0, 4095] = float("inf")
        y = P.ops.linear(xi, pk, sc, None, n, k, 32, out_dtype=torch.float32)
        ref = xi.float() @ wd.t()
        assert torch.equal(torch.isnan(y), torch.isnan(ref))
        assert torch.equal(torch.isposinf(y), torch.isposinf(ref)) and torch.equal(torch.isneginf(y), torch.isneginf(ref))
        fin = torch.isfinite(ref)
        if bool(fin.any()):
            assert float(((y - ref)[fin].abs() / (xi.float().abs() @ wd.abs().t())[fin]).max()) < 1e-5


@pytest.mark.parametrize("m", [1, 4, 16])
def test_power_of_two_scaling_of_activations_is_exact(P, m):
    """Both tensor-core paths rescale activations by powers of two only, so y(2^s x) == 2^s y(x) bit for bit -
    for tiny, huge and mixed magnitudes alike (K = 14336 also runs the partial-sum reduction)."""
    dev = torch.device(DEV)
    for n, k in ((64, 4096), (40, 14336)):
        w = P.ops.generate(n * k, 31, 0.02, torch.float16, dev).view(n, k)
        pk, sc = P.ops.encode(w, 32)
        x = P.ops.generate(m * k, 32 + m, 1.0, torch.bfloat16, dev).view(m, k).clone()
        x[:, ::97] *= 2.0 ** -12                                  # a spread of magnitudes inside every group
        x[:, 5::512] = 0.0
        y = P.ops.linear(x, pk, sc, None, n, k, 32, out_dtype=torch.float32)
        for s in (-80, -30, 40, 90):
            ys = P.ops.linear(x * 2.0 ** s, pk, sc, None, n, k, 32, out_dtype=torch.float32)
            assert torch.equal(ys, y * 2.0 ** s), (m, n, k, s)


def _import_reference():
    """The reference package, from an install under baseline/_ref or a checkout beside this repository."""
    os.environ.setdefault("OJASX_DISABLE_UPDATE_CHECK", "1")
    candidates = [os.environ.get("OJASX_REFERENCE_DIR"), os.path.join(ROOT, "baseline", "_ref"),
                  os.path.join(os.path.dirname(ROOT), "reference")]
    for c in candidates:
        if c and os.path.isdir(os.path.join(c, "ojasx2")):
            if c not in sys.path:
                sys.path.insert(0, c)
            try:
                import logging
                logging.disable(logging.CRITICAL)
                import ojasx2.math.lattice as ref_lattice          # noqa: F401
                return ref_lattice
            except Exception:
                continue
            finally:
                import logging
                logging.disable(logging.NOTSET)
    return None


def test_reference_layer_runs_on_cuda_through_the_patched_seam(P, oracle):
    """install_into_reference() rebinds the module-level dispatcher the reference's forward calls
    (ojasx2/math/lattice.py:51-55,583-589).  The REFERENCE's own E8LatticeLinear then runs on CUDA: with the
    seam its result comes from this library's kernel and must match the result of its stock unpack + F.linear
    path on the same buffers (the check the reference's seam test makes, tests/test_fused_e8_gemm.py:129-150)."""
    ref = _import_reference()
    if ref is None:
        pytest.skip("reference package not importable here")
    dev = torch.device(DEV)
    k, n = 512, 192
    lin = torch.nn.Linear(k, n, bias=True)
    with torch.no_grad():
        lin.weight.copy_(torch.from_numpy(oracle.gen_normal(401, n * k, 0.02).reshape(n, k).copy()))
        lin.bias.copy_(torch.from_numpy(oracle.gen_normal(402, n, 0.1).copy()))
    layer = ref.E8LatticeLinear.from_linear(lin, bitrate=1.5, group_size=32).to(dev)      # packed by the reference on CPU
    ours = P.E8LatticeLinear.from_linear(lin.to(dev), bitrate=1.5, group_size=32)
    assert torch.equal(layer.packed_weight, ours.packed_weight) and torch.equal(layer.block_scales, ours.block_scales)
    calls = []
    stock = ref.dispatch_tilelang_e8_gemm
    try:
        assert P.install_into_reference()

        def spy(*args, **kwargs):
            out = P.dispatch_tilelang_e8_gemm(*args, **kwargs)
            calls.append(out is not None)
            return out

        ref.dispatch_tilelang_e8_gemm = spy
        for m, dt in ((3, torch.bfloat16), (40, torch.bfloat16), (5, torch.float16)):
            x = torch.from_numpy(oracle.gen_normal(403 + m, m * k, 1.0).reshape(m, k).copy()).to(dt).to(dev)
            y_seam = layer(x)
            ref.dispatch_tilelang_e8_gemm = lambda *a, **kw: None               # the reference's own fallback ladder
            y_stock = layer(x)
            ref.dispatch_tilelang_e8_gemm = spy
            assert y_seam.dtype == dt and tuple(y_seam.shape) == (m, n)
            w = layer.unpack_weights(torch.float32)
            exact = x.float() @ w.t() + layer.bias.float()
            assert float((y_seam.float() - exact).norm() / exact.norm()) <= 2e-3
            assert float((y_seam.float() - y_stock.float()).norm() / exact.norm()) <= 6e-3    # stock path rounds W to x's dtype
        assert calls and all(calls)
    finally:
        ref.dispatch_tilelang_e8_gemm = stock


@pytest.mark.parametrize("m,k,n,dt", [(1, 4096, 96, torch.bfloat16), (4, 4096, 96, torch.float16), (8, 1024, 40, torch.bfloat16),
                                      (1, 14336, 64, torch.bfloat16), (5, 14336, 64, torch.float16)])
def test_adapter_term_in_the_decode_epilogue(P, m, k, n, dt):
    """ojx_e8t_gemv_lora: y = x . W^T + bias + lora_t . lora_b in one launch (also through the K > 4096 reduction),
    against the fp32 dense computation; the adapter term of E8LatticeLinear.forward_fused
    (ojasx2/math/lattice.py:839-842)."""
    dev = torch.device(DEV)
    w = P.ops.generate(n * k, 41, 0.02, torch.float16, dev).view(n, k)
    pk, sc = P.ops.encode(w, 32)
    wd = P.ops.decode(pk, sc, (n, k), torch.float32)
    x = P.ops.generate(m * k, 42 + m, 1.0, dt, dev).view(m, k)
    bias = P.ops.generate(n, 43, 0.1, dt, dev)
    r = 8
    t = torch.randn(m, r, device=dev) * 3.0
    b = (torch.randn(r, n, device=dev) * 0.5).to(dt)
    y = P.ops.linear_lora(x, pk, sc, bias, n, k, 32, t, b, out_dtype=torch.float32)
    ref = x.float() @ wd.t() + bias.float() + t @ b.float()
    magnitude = x.float().abs() @ wd.abs().t() + bias.float().abs() + t.abs() @ b.float().abs()
    assert float(((y - ref).abs() / magnitude).max()) < 1e-5
    plain = P.ops.linear(x, pk, sc, bias, n, k, 32, out_dtype=torch.float32)
    assert torch.equal(P.ops.linear_lora(x, pk, sc, bias, n, k, 32, torch.zeros_like(t), b, out_dtype=torch.float32), plain)
    y16 = P.ops.linear_lora(x, pk, sc, None, n, k, 32, t, b)
    assert y16.dtype == dt
    assert float((y16.float() - (ref - bias.float())).abs().max()) <= 2.0 ** -7 * float(ref.abs().max()) + 1e-3


def test_layer_with_adapter_takes_the_fused_epilogue_at_inference(P):
    dev = torch.device(DEV)
    torch.manual_seed(3)
    lin = torch.nn.Linear(1024, 72, bias=True).to(dev).to(torch.bfloat16)
    for had in (False, True):
        layer = P.E8LatticeLinear.from_linear(lin, rank=8, bitrate=1.5, group_size=32, use_hadamard=had)
        with torch.no_grad():
            layer.lora_B.copy_(torch.randn_like(layer.lora_B) * 0.1)
        x = torch.randn(3, 1024, device=dev).to(torch.bfloat16)
        wd = layer.unpack_weights(torch.float32)              # rotated back when the layer stores rotated weights
        ref = (x.float() @ wd.t() + lin.bias.float()
               + layer.scaling * ((x @ layer.lora_A.to(x.dtype)).float() @ layer.lora_B.float()))
        calls = []
        orig = P.ops.linear_lora
        P.ops.linear_lora = lambda *a, **kw: (calls.append(1), orig(*a, **kw))[1]
        try:
            with torch.no_grad():
                y = layer(x)
            assert len(calls) == 1                             # one launch carries the adapter
            y_train = layer(x)                                 # adapters require grad: the differentiable route
            assert len(calls) == 1 and y_train.requires_grad
            with torch.no_grad():
                y9 = layer(torch.randn(9, 1024, device=dev).to(torch.bfloat16))   # more than eight rows: separate term
            assert len(calls) == 1 and y9.shape == (9, 72)
        finally:
            P.ops.linear_lora = orig
        assert float((y.float() - ref).norm() / ref.norm()) < 4e-3
        assert float((y_train.float() - ref).norm() / ref.norm()) < 8e-3
    with pytest.raises(ValueError):
        P.ops.linear_lora(torch.zeros(9, 1024, device=dev, dtype=torch.bfloat16), layer.packed_weight, layer.block_scales,
                          None, 72, 1024, 32, torch.zeros(9, 8, device=dev), torch.zeros(8, 72, device=dev))


@pytest.mark.parametrize("rank,m", [(0, 3), (0, 40), (4, 3)])
def test_traced_layer_computes_with_its_own_input(P, rank, m):
    """torch.jit.trace of a layer without gradients records an operation, not the result for the traced input."""
    dev = torch.device(DEV)
    layer = P.E8LatticeLinear.from_linear(torch.nn.Linear(256, 64).to(dev).bfloat16(), rank=rank, group_size=32, bitrate=1.5).requires_grad_(False)
    if rank:
        layer.lora_B.normal_()
    a, b = torch.randn(m, 256, device=dev).bfloat16(), torch.randn(m, 256, device=dev).bfloat16()
    traced = torch.jit.trace(layer, a, check_trace=False)
    want = layer(b)
    assert float((traced(b).float() - want.float()).norm() / want.float().norm()) <= 1e-2
