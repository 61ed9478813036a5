"""Kernels and dispatch branches at the sizes where they can go wrong: edges of tiles and blocks, remainders, misaligned
rows, the smallest and largest of a branch's range.  Bytes and scales exact against the CPU oracle or the element-wise
chain; float32 solves against float64 with the tolerances of the other GPU tests."""
import pytest
import torch

import oracle
from helpers import args_from, bits_equal, mismatch, synth_acts, synth_weight
from llm_compressor_b200 import GPTQModifier, QuantizationModifier, _lib, compress_state_dict, gptq, modifiers, observers, oneshot, ops
from llm_compressor_b200.awq import scaled_fake_quantize
from llm_compressor_b200.quant_args import QuantizationArgs, preset_name_to_scheme

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(autouse=True, scope="module")
def _leave_the_allocator_as_it_was():
    yield
    torch.cuda.empty_cache()


def _spec(scheme):
    if scheme == "FP8_BLOCK":
        return oracle.preset("FP8_DYNAMIC", strategy="block", block_structure=[128, 128])
    return oracle.preset(scheme)


def _spd(K, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    X = torch.randn(2 * K + 64, K, generator=g, device=DEV, dtype=torch.float64)
    H = X.t() @ X / K
    H.diagonal().add_(0.05)
    return H


def _inverse_residual(U, H):
    """U^T U = H^-1, seen as U H U^T = I (float64, on the device)."""
    U = U.double()
    return float((U @ H @ U.t() - torch.eye(H.shape[0], device=DEV, dtype=torch.float64)).abs().max())


# one, two and three outer blocks of 512, their remainders, odd widths, and tile widths of the products
@pytest.mark.parametrize("K", [1, 16, 127, 129, 511, 512, 513, 640, 1030, 1536, 2500])
def test_factor_at_block_edges(K):
    H = _spd(K, K)
    one = H.float()
    assert ops.gptq_factor(one) == 0
    assert float(one.tril(-1).abs().max()) == 0.0 if K > 1 else True
    assert _inverse_residual(one, H) < 2e-4
    if K <= 1030:
        many = [H.float() for _ in range(3)]
        assert int(ops.gptq_factor_batched(many).abs().max()) == 0
        assert all(_inverse_residual(u, H) < 2e-4 for u in many)


# rows: one CTA, part of one, more CTAs than SMs (narrow superblocks); columns: superblock and micro-block remainders
@pytest.mark.parametrize("N,K,scheme", [(1, 16, "FP8_DYNAMIC"), (33, 520, "FP8_DYNAMIC"), (64, 1032, "W8A16"),
                                        (31, 513, "W8A16"), (4768, 264, "FP8_DYNAMIC"), (5000, 640, "W4A16")])
def test_sweep_at_superblock_edges(N, K, scheme):
    args = preset_name_to_scheme(scheme, ["Linear"]).weights
    w = (torch.randn(N, K, generator=torch.Generator().manual_seed(K)) * 0.02).bfloat16().to(DEV)
    H = _spd(K, 3)
    U = torch.linalg.cholesky(torch.linalg.inv(H), upper=True).contiguous()
    scale, zp = ops.qparams(*ops.observe_minmax(w, args), args)
    wf = w.float()
    losses = ops.gptq_sweep(wf, U.float(), scale, None, args)
    # the recursion in float64 with the same codes' rules, column by column
    ref, Ud = w.double(), U
    spread = scale.float() if scale.shape[1] == 1 else scale.float().repeat_interleave(args.group_size, 1)
    qmin, qmax = (-448.0, 448.0) if args.type == "float" else (-(1 << (args.num_bits - 1)), (1 << (args.num_bits - 1)) - 1)
    out, total = torch.empty_like(wf), torch.zeros(N, device=DEV, dtype=torch.float64)
    for i in range(K):
        s = spread[:, min(i, spread.shape[1] - 1)]
        v = (ref[:, i].float() / s).clamp(qmin, qmax)
        q = v.to(torch.float8_e4m3fn).float() if args.type == "float" else v.round()
        q = (q * s).bfloat16().float()
        err = (ref[:, i] - q.double()) / Ud[i, i]
        out[:, i], total = q, total + err * err / 2
        ref[:, i + 1:] -= err[:, None] * Ud[i, i + 1:]
    assert mismatch(wf, out) <= 0.005
    assert torch.allclose(losses.double(), total, rtol=0.02, atol=1e-9)


def test_sweep_exact_pass_at_rounding_boundaries():
    """Every quotient on a rounding boundary: the fast test of a code fails in every micro-block."""
    args = preset_name_to_scheme("W8A16", ["Linear"]).weights
    N, K = 40, 96
    w = (torch.randint(-100, 100, (N, K), generator=torch.Generator().manual_seed(0)).float() + 0.5) * 0.0078125
    wf = w.to(DEV)
    scale = torch.full((N, 1), 0.0078125, device=DEV).bfloat16()
    ops.gptq_sweep(wf, None, scale, None, args)
    assert bits_equal(wf, (w / 0.0078125).round() * 0.0078125)


@pytest.mark.parametrize("count,N,K,scheme", [(5, 96, 520, "FP8_DYNAMIC"), (3, 70, 640, "W4A16")])
def test_batched_sweep_with_shared_factors(count, N, K, scheme):
    args = preset_name_to_scheme(scheme, ["Linear"]).weights
    Us = [torch.linalg.cholesky(torch.linalg.inv(_spd(K, i)), upper=True).float().contiguous() for i in range(2)]
    pick = [Us[i % 2] for i in range(count)]
    ws = [(torch.randn(N, K, generator=torch.Generator().manual_seed(i)) * 0.02).bfloat16().to(DEV) for i in range(count)]
    qp = [ops.qparams(*ops.observe_minmax(w, args), args) for w in ws]
    got = [w.float() for w in ws]
    losses = ops.gptq_sweep_batched(got, pick, [s for s, _ in qp], None, args)
    for k in range(count):
        ref = ws[k].float()
        ref_losses = ops.gptq_sweep(ref, pick[k], qp[k][0], None, args)
        assert mismatch(got[k], ref) <= 0.005
        assert torch.allclose(losses[k], ref_losses, rtol=0.01)


# columns in order and permuted, whole 16-byte pieces and not, rows that are no multiple of four, K too wide for four
# rows in shared memory
@pytest.mark.parametrize("N,K", [(1, 1), (3, 40), (5, 37), (130, 1160), (2, 30000)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_column_gathers_and_scatters(N, K, dtype):
    g = torch.Generator(device=DEV).manual_seed(K)
    w = torch.randn(N, K, generator=g, device=DEV).to(dtype)
    perm = torch.randperm(K, generator=g, device=DEV).int()
    diag = (torch.rand(K, generator=g, device=DEV) > 0.3).float()
    for p in (None, perm):
        ref = w.float() if p is None else w.float()[:, p.long()]
        assert torch.equal(ops.gather_columns_f32(w, p), ref)
        assert torch.equal(ops.scatter_columns_cast(ref, dtype, p), w)
        ws = [w, w.flip(0).contiguous()]
        many = ops.gather_columns_f32_batched(ws, None if p is None else [p, p], [diag, diag])
        assert torch.equal(many[0], ref * diag)
        back = ops.scatter_columns_cast_batched(torch.stack([ref, ref]), dtype, None if p is None else [p, p])
        assert torch.equal(back[1], w)


@pytest.mark.parametrize("K", [3, 40, 129, 700])
def test_batched_prologue_and_mirror(K):
    Hs = [torch.randn(K, K, generator=torch.Generator(device=DEV).manual_seed(i), device=DEV) for i in range(3)]
    for H in Hs:
        H.diagonal().abs_()
        H[K // 2, K // 2] = 0.0   # a dead column
    full = [H.clone() for H in Hs]
    ops.hessian_finalize_many(full, [0.5, 1.0, 2.0])
    for H, f, s in zip(Hs, full, (0.5, 1.0, 2.0)):
        one = H.clone()
        ops.hessian_finalize(one, s)
        low = (H * s).tril()
        assert torch.equal(f, low + low.tril(-1).t()) and torch.equal(f, one)
    for actorder in (False, True):
        mats, perm, diag = ops.gptq_prologue_batched([f.clone() for f in full], 0.01, actorder)
        for i, f in enumerate(full):
            H, p, d = gptq._factor_prologue(f.clone(), 0.01, "weight" if actorder else None)
            assert torch.equal(diag[i], d)
            assert not actorder or torch.equal(perm[i], p)
            assert torch.allclose(mats[i], H, rtol=1e-6, atol=0)


# short and long accumulation, widths with a ragged last tile, one split and many
@pytest.mark.parametrize("T,K", [(8, 8), (64, 264), (513, 1160), (1024, 4104), (2048, 2056)])
def test_hessian_update_adds_to_what_is_there(T, K):
    g = torch.Generator(device=DEV).manual_seed(T)
    xs = [torch.randn(T, K, generator=g, device=DEV).bfloat16() for _ in range(2)]
    H = torch.zeros(K, K, device=DEV)
    for x in xs:
        ops.hessian_syrk(x, H)
    ops.hessian_finalize(H, 0.5)
    ref = sum(x.double().t() @ x.double() for x in xs)
    assert float((H.double() - ref).norm() / ref.norm()) < 1e-5


SCHEMES = ["W4A16", "W4A16_ASYM", "W8A16", "FP8_DYNAMIC", "FP8_BLOCK", "NVFP4A16", "MXFP4A16", "MXFP8A16"]


# a row or block each per warp, lane or CTA; ragged blocks; rows misaligned to 16 bytes; too many rows for a CTA each
@pytest.mark.parametrize("scheme", SCHEMES)
@pytest.mark.parametrize("N,K", [(3, 128), (130, 384), (129, 1152), (2400, 256), (67, 200)])
def test_one_pass_parameters_and_codes(scheme, N, K):
    s = preset_name_to_scheme(scheme, ["Linear"])
    args = s.weights
    if args.group_size and K % args.group_size:
        pytest.skip("group size does not divide K")
    names = ["gate_proj", "up_proj"] if scheme == "NVFP4A16" else ["o_proj"]
    model = torch.nn.Module()
    for i, name in enumerate(names):
        lin = torch.nn.Linear(K, N, bias=False, dtype=torch.bfloat16, device=DEV)
        lin.weight.data = (synth_weight(N, K, seed=N + K + i) * (1 + 3 * i)).to(DEV)
        model.add_module(name, lin)
    oneshot(model, recipe=QuantizationModifier(targets="Linear", scheme=scheme))
    spec = _spec(scheme)
    obs = [oracle.WeightObserver(spec) for _ in names]
    if len(obs) > 1:
        top = max(float(model.get_submodule(n).weight.data.abs().max()) for n in names)
    for name, o in zip(names, obs):
        lin = model.get_submodule(name)
        w = lin.weight.data.cpu()
        if len(obs) > 1:   # the global scale of the larger of the two: an element of that size in a copy of the weight
            lift = torch.cat([w, torch.full((1, K), top, dtype=w.dtype)])
            qp = o(lift).get_qparams()
            qp = dict(qp, scale=qp["scale"][:N], zero_point=qp["zero_point"][:N])
            assert bits_equal(lin.weight_global_scale.data, qp["global_scale"])
        else:
            qp = o(w).get_qparams()
        assert bits_equal(lin.weight_scale.data, qp["scale"].to(w.dtype))
        assert bits_equal(lin.weight_zero_point.data, qp["zero_point"])
        sd = {"weight": w, "weight_scale": qp["scale"].to(w.dtype), "weight_zero_point": qp["zero_point"]}
        if qp["global_scale"] is not None:
            sd["weight_global_scale"] = qp["global_scale"]
        ref = oracle.compress_weight(sd, spec)
        out = compress_state_dict({k: v.to(DEV) for k, v in sd.items()}, s, "pack-quantized" if args.type == "int" else None)
        for k in ("weight_packed", "weight"):
            if k in ref and k in out:
                assert bits_equal(out[k], ref[k]), (k, mismatch(out[k], ref[k]))


def test_batched_parameters_equal_the_single_ones():
    for scheme in ("W4A16_ASYM", "W8A16", "FP8_BLOCK", "MXFP4A16"):
        args = preset_name_to_scheme(scheme, ["Linear"]).weights
        ws = [synth_weight(200, 256, seed=i).to(DEV) for i in range(5)]
        scales, zps = ops.minmax_qparams(ws, args)
        for w, s, z in zip(ws, scales, zps):
            ref_s, ref_z = ops.qparams(*ops.observe_minmax(w, args), args)
            assert bits_equal(s, ref_s) and bits_equal(z, ref_z)


# groups and channels, symmetric or not, odd rows, channels of one and of many pieces per lane
@pytest.mark.parametrize("kw", [dict(num_bits=4, symmetric=True, strategy="group", group_size=128),
                                dict(num_bits=4, symmetric=False, strategy="group", group_size=32),
                                dict(num_bits=8, symmetric=False, strategy="channel"),
                                dict(num_bits=8, symmetric=True, strategy="channel")])
@pytest.mark.parametrize("N,K", [(3, 128), (33, 384), (7, 4096), (130, 6144)])
def test_scale_search_step_equals_the_element_wise_chain(kw, N, K):
    args = QuantizationArgs(type="int", **kw)
    w = synth_weight(N, K, seed=N + K).to(DEV)
    s = torch.exp(0.5 * torch.randn(K, generator=torch.Generator(device=DEV).manual_seed(1), device=DEV))
    got = ops.scaled_fake_quantize(w, s, args)
    assert got is not None
    scaled = (w * s.view(1, -1)).to(w.dtype)
    qp = ops.qparams(*ops.observe_minmax(scaled, args), args)
    ref = (ops.fake_quantize(scaled, qp[0], qp[1], args) / s.view(1, -1)).to(w.dtype)
    assert bits_equal(got, ref), mismatch(got, ref)


# more weights than a launch takes, of different heights and strides, one and two chunks a lane, a part of a warp's columns
@pytest.mark.parametrize("g,K", [(8, 264), (16, 48), (128, 1152), (256, 512)])
def test_scale_search_step_of_many_weights(g, K):
    args = QuantizationArgs(num_bits=4, type="int", symmetric=False, strategy="group", group_size=g)
    ws = [synth_weight(200, K + 8 * (n % 2), seed=n).to(DEV)[-n:, :K] for n in (1, 33, 8, 200, 7, 64, 3, 9, 17)]
    s = torch.exp(0.5 * torch.randn(K, generator=torch.Generator(device=DEV).manual_seed(1), device=DEV))
    got = ops.scaled_fake_quantize_many(ws, s, args)
    for w, out in zip(ws, got):
        scaled = (w * s.view(1, -1)).to(w.dtype)
        qp = ops.qparams(*ops.observe_minmax(scaled, args), args)
        assert bits_equal(out, (ops.fake_quantize(scaled, qp[0], qp[1], args) / s.view(1, -1)).to(w.dtype))


# table of powers: every code type, groups and whole rows, symmetric or not, rows that are no multiple of a CTA's
@pytest.mark.parametrize("scheme", SCHEMES)
@pytest.mark.parametrize("N,K", [(3, 128), (130, 640)])
def test_grid_search_against_the_oracle(scheme, N, K):
    args = preset_name_to_scheme(scheme, ["Linear"]).weights
    w = synth_weight(N, K, seed=5 * N + K)
    spec = _spec(scheme)
    o = oracle.WeightObserver(spec, "memoryless_mse")
    o(w)
    mn, mx = ops.observe_mse(w.to(DEV), args)
    # two candidates whose errors are equal to rounding may swap: compare all but a few groups
    for got, ref in ((mn, o.min_vals), (mx, o.max_vals)):
        differ = (got.cpu().float() != ref.float()).float().mean()
        assert float(differ) <= 0.02, float(differ)
        assert float((got.cpu().float() - ref.float()).norm() / ref.float().norm()) < 0.02


def test_a_solve_that_raises_leaves_the_others_quantised():
    parent = torch.nn.Module()
    for k in range(3):
        lin = torch.nn.Linear(256, 64, bias=False, device=DEV, dtype=torch.bfloat16)
        lin.weight.data = synth_weight(64, 256, k).to(DEV)
        parent.add_module(f"p{k}", lin)
    mod = GPTQModifier(targets="Linear", scheme="W4A16", actorder=None)
    mod.on_initialize(parent)
    mod.on_calibration_start(parent)
    for k, lin in enumerate(parent.children()):
        mod.calibrate_module(lin, (synth_acts(2, 512, 256, k).to(DEV),), None)
    before = [lin.weight.data.clone() for lin in parent.children()]

    class Broken(observers.MemorylessMinMaxObserver):
        def update_statistics_from_weight(self, weight):
            raise RuntimeError("no statistics today")
    parent.p0.weight_observer = Broken("weight", parent.p0.quantization_scheme.weights)
    with pytest.raises(RuntimeError, match="no statistics today"):
        mod.on_sequential_epoch_end(parent, list(parent.modules()))
    assert torch.equal(parent.p0.weight.data, before[0]) and parent.p0.quantization_status != "frozen"
    for k in (1, 2):
        lin = getattr(parent, f"p{k}")
        assert not torch.equal(lin.weight.data, before[k]) and lin.quantization_status == "frozen"
    assert sorted(mod.losses) == ["p1", "p2"]


@pytest.mark.parametrize("many", [False, True])
def test_status_word_does_not_keep_the_hessian(many):
    K = 1024
    lin = torch.nn.Linear(K, 8, bias=False, device=DEV, dtype=torch.bfloat16)
    groups = [modifiers._HessianGroup(lin) for _ in range(2)]
    for g in groups:
        g.accumulate(synth_acts(1, 256, K, 0).to(DEV))
        g.flush()
    if many:
        modifiers._finalize_groups(groups)
    Hs = [g.finalized() for g in groups]
    before = torch.cuda.memory_allocated()
    del Hs
    assert torch.cuda.memory_allocated() <= before - 2 * 4 * K * K
    assert [int(g.status) for g in groups] == [0, 0]


# pivots below the smallest normal float32 (1.2e-38): alone, and one among normal ones in the middle of a 16-column step
@pytest.mark.parametrize("K,tiny", [(1, [0]), (16, range(16)), (130, range(130)), (200, [77])])
def test_factor_accepts_subnormal_pivots(K, tiny):
    d = torch.full((K,), 4.0, dtype=torch.float64)
    for i in tiny:
        d[i] = 1e-39 * (1 + i % 7)
    H = torch.diag(d).float().to(DEV)
    ref = 1.0 / H.diagonal().double().sqrt()
    many = [H.clone() for _ in range(2)]
    assert ops.gptq_factor(H) == 0
    assert int(ops.gptq_factor_batched(many).abs().max()) == 0
    for U in [H] + many:
        assert torch.allclose(U.diagonal().double(), ref, rtol=2e-7)
        assert float((U - torch.diag(U.diagonal())).abs().max()) == 0.0


@pytest.mark.parametrize("K,column,value", [(16, 3, 0.0), (200, 150, -1e-39), (200, 77, float("nan")), (640, 600, -0.0)])
def test_factor_reports_the_first_bad_pivot(K, column, value):
    H = torch.diag(torch.full((K,), 4.0)).to(DEV)
    H[column, column] = value
    status = ops.gptq_factor_async(H).tolist()
    assert status == [_lib.NOT_POSITIVE_DEFINITE, K - column, 0, 0]   # (columns are counted in reversed order)


@pytest.mark.parametrize("scheme", ["W4A16", "W4A16_ASYM", "W8A16", "FP8_DYNAMIC", "FP8_BLOCK", "MXFP4A16", "MXFP8A16"])
@pytest.mark.parametrize("N,K", [(8, 2048), (2400, 384), (130, 256)])
def test_one_launch_parameters_of_unusual_values(scheme, N, K):
    """Statistics and parameters in one launch leave a NaN of either sign out as the two launches do."""
    args = preset_name_to_scheme(scheme, ["Linear"]).weights
    w = synth_weight(N, K, seed=N + K)
    nan, inf = float("nan"), float("inf")
    for row, col, value in ((1, 5, nan), (2, 6, -nan), (3, K - 1, -nan), (4, 0, inf), (5, 7, -inf), (6, 9, 3.3e38), (6, 10, nan)):
        w[row, col] = value
    w[0, 16:180] = -nan
    w[7] = torch.where(w[7] > 0, torch.tensor(-0.0, dtype=w.dtype), w[7])
    w = w.to(DEV)
    scale, zp = ops.qparams(*ops.observe_minmax(w, args), args)
    one = ops.minmax_qparams(w, args)
    many = ops.minmax_qparams([w.clone(), w], args)
    for s, z in (one, (many[0][0], many[1][0]), (many[0][1], many[1][1])):
        assert bits_equal(s, scale) and bits_equal(z, zp)


@pytest.mark.parametrize("N,K", [(1, 1), (31, 7), (33, 17), (64, 47), (65, 49), (32, 129), (40, 511), (33, 520),
                                 (4736, 40), (4737, 136), (4801, 264)])
@pytest.mark.parametrize("scheme", ["W8_CHANNEL", "W4_ASYM"])
def test_sweep_at_edges_of_blocks(N, K, scheme):
    """Half-blocks of 8 columns, operands of 16, tiles of 128, superblocks of 512 (32 rows a CTA) and 256 (64)."""
    g = torch.Generator().manual_seed(N * 1000 + K)
    a = torch.randn(3 * K + 8, K, generator=g, dtype=torch.float64)
    U = torch.linalg.cholesky(torch.linalg.inv(a.T @ a / len(a) + 0.05 * torch.eye(K, dtype=torch.float64)), upper=True)
    w = (torch.randn(N, K, generator=g) * 0.02).to(torch.float64)
    asym = scheme == "W4_ASYM"
    scale = torch.full((N, 1), 0.01 if asym else 5e-4).bfloat16()
    zp = (torch.arange(N) % 5 - 2).to(torch.int8).view(N, 1) if asym else None
    args = QuantizationArgs(num_bits=4 if asym else 8, type="int", symmetric=not asym, strategy="channel")
    lo, hi = (-8, 7) if asym else (-128, 127)
    x, s, z = w.clone(), scale.double(), zp.double() if asym else torch.zeros(N, 1, dtype=torch.float64)
    q, loss, close = torch.zeros_like(w), torch.zeros(N, dtype=torch.float64), torch.zeros(N, dtype=torch.bool)
    for i in range(K):
        v = x[:, i:i + 1] / s + z
        c = v.clamp(lo, hi)
        # float32 sums (errors below 1e-6 of the weights' size) may turn a code this close to a boundary, and with it
        # everything later in the row
        close |= ((c - c.floor() - 0.5).abs() < 1e-3)[:, 0]
        q[:, i] = ((c.round() - z) * s).bfloat16().double()[:, 0]
        e = (x[:, i] - q[:, i]) / U[i, i]
        loss += e * e / 2
        x[:, i:] -= e[:, None] * U[i, i:]
    W = w.float().cuda()
    losses = ops.gptq_sweep(W, U.float().cuda().contiguous(), scale.cuda(), None if zp is None else zp.cuda(), args)
    torch.cuda.synchronize()
    sure = ~close
    assert torch.equal(W.cpu().double()[sure], q[sure])
    assert torch.allclose(losses.cpu().double()[sure], loss[sure], rtol=1e-4)
    assert float((W.cpu().double() != q).double().mean()) < 0.05


@pytest.mark.parametrize("K", [640, 1100, 1664])
def test_factor_and_sweep_of_badly_scaled_problems(K):
    """Operands of halves have a scale per row: columns 2^40 apart in size give the factor and the codes of equal ones."""
    H = _spd(K, K).float()
    e = torch.randint(-20, 21, (K,), generator=torch.Generator().manual_seed(K)).to(DEV)
    s = torch.ldexp(torch.ones(K, device=DEV), e)
    U, V = H.clone(), H * s[:, None] * s[None, :]
    assert ops.gptq_factor(U) == 0 and ops.gptq_factor(V) == 0
    W = V * s[None, :]   # (S H S)^-1 = S^-1 U^T U S^-1
    ref = torch.linalg.cholesky(torch.linalg.inv(H.double()), upper=True)
    for got in (U, W):   # float32 at this conditioning: about 1e-6
        assert float((torch.triu(got).double() - ref).norm() / ref.norm()) < 5e-6
    w = torch.randn(96, K, generator=torch.Generator().manual_seed(1)).to(DEV)
    scale = torch.full((96, 1), 0.5, device=DEV).bfloat16()
    args = QuantizationArgs(num_bits=8, type="int", strategy="channel")
    a, b = w.clone(), w.clone()
    ops.gptq_sweep(a, torch.triu(U).contiguous(), scale, None, args)
    # rows of U scaled alike scale the errors inversely and leave the corrections as they are
    ops.gptq_sweep(b, (torch.triu(U) * s[:, None]).contiguous(), scale, None, args)
    assert mismatch(a, b) < 0.005


@pytest.mark.parametrize("N,K", [(64, 1024), (64, 4096), (4736, 1024), (4736, 4096)])
def test_concurrent_sweeps_read_nothing_before_it_is_written(N, K):
    """Superblocks' operands are made on helper streams: one problem alone and as one of nine that crowd the GPU, each on a
    stream of its own with a workspace of NaN, give the same bits."""
    lib, count = _lib.load(), 9
    g = torch.Generator(device=DEV).manual_seed(N + K)
    U = torch.triu(torch.randn(K, K, generator=g, device=DEV) / K ** 0.5, 1)
    U.diagonal().copy_(torch.exp2(torch.randint(-3, 4, (K,), generator=g, device=DEV).float()))
    w = torch.randn(N, K, generator=g, device=DEV) * 0.02
    scale = torch.full((N, 1), 5e-4, device=DEV).bfloat16()
    args = QuantizationArgs(num_bits=8, type="int", strategy="channel")

    def problem():
        ws = torch.full((lib.b200q_gptq_sweep_workspace_bytes(N, K, 128),), 0xFF, dtype=torch.uint8, device=DEV)
        return w.clone(), torch.empty(N, device=DEV), ws

    def run(W, losses, ws):
        _lib.check(lib.b200q_gptq_sweep(W.data_ptr(), N, K, K, U.data_ptr(), K, scale.data_ptr(), _lib.BF16, None, None, None,
                                        args.c_struct(), 128, losses.data_ptr(), ws.data_ptr(), _lib.stream_ptr()), "sweep")

    alone, many = problem(), [problem() for _ in range(count)]
    run(*alone)
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(count)]
    for stream, p in zip(streams, many):
        with torch.cuda.stream(stream):
            run(*p)
    torch.cuda.synchronize()
    assert bool(torch.isfinite(alone[1]).all()) and int(alone[2][:4].view(torch.int32)) == 0
    for W, losses, ws in many:
        assert bits_equal(W, alone[0]) and bits_equal(losses, alone[1]) and int(ws[:4].view(torch.int32)) == 0


def test_a_sum_taken_on_another_stream_is_not_given_out_before_it_is_read():
    K, tokens = 1536, 2048
    lin = torch.nn.Linear(K, 8, bias=False, device=DEV, dtype=torch.bfloat16)
    torch.cuda.empty_cache()
    x = torch.randn(1, 64, K, device=DEV).bfloat16()
    modifiers._HessianGroup(lin).accumulate(x)   # (loads the kernels)
    torch.cuda.synchronize()
    group = modifiers._HessianGroup(lin, stage_tokens=tokens)
    group.accumulate(x)
    taken = [(t.untyped_storage().data_ptr(), t.untyped_storage().nbytes()) for t in (group.H, group._stage)]
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        torch.cuda._sleep(200_000_000)   # (about a tenth of a second, the readers behind it)
        group.take_sum()                 # (and dropped)
    given = [torch.empty(n, dtype=torch.uint8, device=DEV) for _, n in taken]
    assert not stream.query()
    for (at, n), t in zip(taken, given):
        assert all(t.data_ptr() >= a + m or t.data_ptr() + t.nbytes <= a for a, m in taken)
    torch.cuda.synchronize()
