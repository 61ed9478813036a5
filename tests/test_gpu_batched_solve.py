"""Batched solve of many small problems (b200q_gptq_factor_batched, b200q_gptq_sweep_batched and
the GPTQModifier path that uses them) against float64, the single-problem kernels and the CPU
oracle.  Same tolerances as the single-problem tests: factors within a small multiple of the
float32 chain's own error, GPTQ weights with at least 99.5 % identical values, identical scales,
loss within 1 %."""
import warnings

import pytest
import torch

import oracle
from helpers import args_from, bits_equal, mismatch, synth_acts, synth_weight
from llm_compressor_b200 import GPTQModifier, _lib, gptq, observers, ops
from test_oracle_golden import spec_from

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
CODE_MATCH = 0.995
LOSS_RTOL = 0.01


def _spd(K, seed):
    g = torch.Generator().manual_seed(seed)
    X = torch.randn(4 * K, K, generator=g) * (0.25 + 2 * torch.rand(K, generator=g))
    H = (2 * X.t() @ X / 4).float()
    H[torch.arange(K), torch.arange(K)] += 0.01 * H.diag().mean()
    return H


@pytest.mark.parametrize("K,count", [(32, 3), (128, 5), (130, 2), (200, 4), (768, 6), (1000, 2), (2048, 2)])
def test_batched_factor_matches_float64(K, count):
    Hs = [_spd(K, 100 * K + i) for i in range(count)]
    dev = [H.clone().to(DEV) for H in Hs]
    status = ops.gptq_factor_batched(dev).cpu()
    assert int(status.abs().max()) == 0
    for H, Hg in zip(Hs, dev):
        Hd = H.double()
        U_ref = torch.linalg.cholesky(torch.cholesky_inverse(torch.linalg.cholesky(Hd)), upper=True)
        U = Hg.cpu().double()
        assert float(U.tril(-1).abs().max()) == 0.0
        err = float((U - U_ref).norm() / U_ref.norm())
        U32 = torch.linalg.cholesky(torch.cholesky_inverse(torch.linalg.cholesky(H.clone())), upper=True).double()
        err32 = float((U32 - U_ref).norm() / U_ref.norm())
        assert err < max(5e-5, 4 * err32), (err, err32)


def test_batched_factor_agrees_with_the_single_problem_kernel():
    K = 640
    Hs = [_spd(K, 7 + i).to(DEV) for i in range(3)]
    single = [H.clone() for H in Hs]
    for H in single:
        assert ops.gptq_factor(H) == 0
    ops.gptq_factor_batched(Hs)
    for a, b in zip(Hs, single):
        assert float((a - b).norm() / b.norm()) < 2e-5


def test_batched_factor_reports_the_failing_problem_only():
    K = 256
    Hs = [_spd(K, i) for i in range(4)]
    Hs[2][200, 200] = -5.0
    dev = [H.clone().to(DEV) for H in Hs]
    status = ops.gptq_factor_batched(dev).cpu()
    assert status[:, 0].tolist() == [0, 0, 1, 0]
    # reversed column order: column 200 of H is column K - 1 - 200 of the factored matrix
    assert int(status[2, 1]) == K - 1 - 200 + 1
    U_ref = torch.linalg.cholesky(torch.cholesky_inverse(torch.linalg.cholesky(Hs[3].double())), upper=True)
    assert float((dev[3].cpu().double() - U_ref).norm() / U_ref.norm()) < 5e-5


def _problem(N, K, seed, tokens_factor=2):
    w = synth_weight(N, K, seed=seed)
    S = min(K // 2, 512)
    x = synth_acts(max(8, -(-tokens_factor * K // S)), S, K, seed=seed + 1)
    H, n = oracle.accumulate_hessian(x, oracle.make_empty_hessian(K), 0)
    return w, H / n


def _lin(w, args):
    N, K = w.shape
    lin = torch.nn.Linear(K, N, bias=False, device=DEV, dtype=w.dtype)
    lin.weight.data = w.to(DEV)
    lin.weight_observer = observers.Observer.load_from_registry(args.observer, base_name="weight", args=args)
    lin.weight_observer(lin.weight.data)
    return lin


SCHEMES = {
    "W4A16": dict(num_bits=4, type="int", symmetric=True, strategy="group", group_size=128),
    "W4A16_ASYM": dict(num_bits=4, type="int", symmetric=False, strategy="group", group_size=128),
    "W8_CHANNEL": dict(num_bits=8, type="int", symmetric=True, strategy="channel"),
    "W4_ACTORDER_WEIGHT": dict(num_bits=4, type="int", symmetric=True, strategy="group", group_size=128,
                               actorder="weight"),
    "W4_ACTORDER_GROUP": dict(num_bits=4, type="int", symmetric=True, strategy="group", group_size=128,
                              actorder="group"),
}


@pytest.mark.parametrize("N,K,scheme,count", [(96, 256, "W4A16", 3), (200, 768, "W4A16", 3), (128, 640, "W4A16_ASYM", 2),
                                              (130, 384, "W8_CHANNEL", 2), (64, 1152, "W4_ACTORDER_WEIGHT", 2),
                                              (64, 512, "W4_ACTORDER_GROUP", 2), (300, 2048, "W4A16", 2)])
def test_batched_gptq_vs_oracle(N, K, scheme, count):
    args = args_from(SCHEMES[scheme])
    problems = [_problem(N, K, seed=31 * N + K + 5 * i) for i in range(count)]
    mods = [_lin(w, args) for w, _ in problems]
    factors = gptq.factor_hessians_batched([H.clone().to(DEV) for _, H in problems], 0.01, args.actorder)
    done = gptq.quantize_weights_batched(mods, args, factors)
    gptq.resolve_factors(factors)
    assert all(f.ok for f in factors)
    for (w, H), (loss, out) in zip(problems, done):
        loss_ref, ref = oracle.quantize_weight(w, _oracle_spec(scheme), H.clone())
        assert bits_equal(out["weight_scale"], ref["weight_scale"])
        assert bits_equal(out["weight_zero_point"], ref["weight_zero_point"])
        if "weight_g_idx" in ref:
            assert torch.equal(out["weight_g_idx"].cpu().long(), ref["weight_g_idx"].long())
        mm = mismatch(out["weight"], ref["weight"])
        assert mm <= 1 - CODE_MATCH, mm
        assert float(loss) == pytest.approx(loss_ref, rel=LOSS_RTOL)


def _oracle_spec(scheme):
    return spec_from(dict(SCHEMES[scheme]))


def test_batched_sweep_agrees_with_the_single_problem_kernel():
    N, K = 160, 896
    args = args_from(SCHEMES["W4A16"])
    problems = [_problem(N, K, seed=11 + i) for i in range(3)]
    single = []
    for w, H in problems:
        lin = _lin(w, args)
        single.append(gptq.quantize_weight(lin, args, H.clone().to(DEV)))
    mods = [_lin(w, args) for w, _ in problems]
    factors = gptq.factor_hessians_batched([H.clone().to(DEV) for _, H in problems], 0.01, None)
    done = gptq.quantize_weights_batched(mods, args, factors)
    for (loss_a, a), (loss_b, b) in zip(done, single):
        assert bits_equal(a["weight_scale"], b["weight_scale"])
        assert mismatch(a["weight"], b["weight"]) <= 1 - CODE_MATCH
        assert float(loss_a) == pytest.approx(loss_b, rel=LOSS_RTOL)


def test_batched_sweep_without_factor_equals_the_single_problem_fallback():
    # no factor: the identity stands in for U (round to nearest); no trailing update runs, so the
    # two kernels must agree bit for bit
    N, K = 70, 256
    args = args_from(SCHEMES["W4A16"])
    ws = [synth_weight(N, K, seed=i) for i in range(2)]
    mods = [_lin(w, args) for w in ws]
    wf = [ops.gather_columns_f32(m.weight.data) for m in mods]
    qp = [m.weight_observer.get_qparams() for m in mods]
    losses = ops.gptq_sweep_batched(wf, None, [q["scale"] for q in qp], [q["zero_point"] for q in qp], args)
    for i, (m, f, q) in enumerate(zip(mods, wf, qp)):
        ref = ops.gather_columns_f32(m.weight.data)
        ref_losses = ops.gptq_sweep(ref, None, q["scale"], q["zero_point"], args)
        assert torch.equal(f, ref)
        assert torch.allclose(losses[i], ref_losses, rtol=1e-5, atol=0)


class _Experts(torch.nn.Module):
    def __init__(self, count, hidden, inter):
        super().__init__()
        g = torch.Generator().manual_seed(0)
        self.up = torch.nn.ModuleList(torch.nn.Linear(hidden, inter, bias=False) for _ in range(count))
        self.down = torch.nn.ModuleList(torch.nn.Linear(inter, hidden, bias=False) for _ in range(count))
        for m in list(self.up) + list(self.down):
            m.weight.data = torch.randn(m.weight.shape, generator=g) * 0.05

    def forward(self, x):
        # every expert sees its own slice of the tokens
        parts = x.chunk(len(self.up), dim=1)
        return torch.cat([d(torch.nn.functional.silu(u(p))) for u, d, p in zip(self.up, self.down, parts)], dim=1)


@pytest.mark.parametrize("fail_one", [False, True])
def test_modifier_takes_the_batched_path_for_many_small_hessians(fail_one):
    count, hidden, inter = 6, 256, 384
    torch.manual_seed(0)
    x = (torch.randn(4, count * 640, hidden) * (0.5 + torch.rand(hidden))).to(torch.bfloat16).to(DEV)

    def run(batch):
        model = _Experts(count, hidden, inter).to(torch.bfloat16).to(DEV)
        mod = GPTQModifier(targets="Linear", scheme="W4A16", batch_small_hessians=batch)
        events = []
        mod.trace = lambda e, m=None: events.append(e)
        mod.on_initialize(model)
        mod.on_calibration_start(model)
        with torch.no_grad():
            model(x)
        if fail_one:
            g = mod._groups[model.up[2]]
            g.flush()
            g.H.zero_()
            g.H.diagonal().fill_(1.0)
            g.H[3, 3] = -4.0
        with warnings.catch_warnings(record=True) as caught:
            warnings.simplefilter("always")
            mod.on_sequential_epoch_end(model, list(model.up) + list(model.down))
        mod.on_calibration_end(model)
        mod.on_finalize(model)
        return model, mod, events, [str(w.message) for w in caught]

    base_model, base, base_events, base_warn = run(0)
    model, mod, events, warned = run(4)
    # one factor event per Hessian either way; the batched run raises them before any sweep
    assert events.count("job_factored") == 2 * count
    assert events.count("job_start") == 1 and base_events.count("job_start") == 2 * count
    assert any("round-to-nearest" in w for w in warned) == fail_one
    assert any("round-to-nearest" in w for w in base_warn) == fail_one
    for (name, a), (_, b) in zip(model.named_modules(), base_model.named_modules()):
        if not isinstance(a, torch.nn.Linear):
            continue
        assert a.quantization_status == "frozen"
        assert bits_equal(a.weight_scale, b.weight_scale)
        assert mismatch(a.weight.data, b.weight.data) <= 1 - CODE_MATCH, name
    for name, loss in mod.losses.items():
        assert loss == pytest.approx(base.losses[name], rel=LOSS_RTOL, abs=1e-9), name


def _spd_factor64(K, tokens):
    """(H as a calibration of so many tokens leaves it, damped; its factor in float64)"""
    g = torch.Generator(device=DEV).manual_seed(K + tokens)
    scale = 0.25 + 2.0 * torch.rand(K, generator=g, device=DEV)
    H = torch.zeros(K, K, device=DEV, dtype=torch.float64)
    for t in range(0, tokens, 4096):
        x = (torch.randn(min(4096, tokens - t), K, generator=g, device=DEV) * scale).bfloat16().double()
        H.addmm_(x.t(), x, alpha=2.0)
    H = H.float()
    H.diagonal().add_(0.01 * H.diagonal().mean())
    L = torch.linalg.cholesky(H.double().flip(0, 1))
    return H, torch.linalg.solve_triangular(L, torch.eye(K, device=DEV, dtype=torch.float64), upper=False).flip(0, 1)


# `limit`: the same error of an elimination by float32 multiply-adds, one thread block a problem (relative, 2-norm)
@pytest.mark.parametrize("K,tokens,limit", [(256, 600, 2.4e-7), (520, 1500, 1.9e-7), (768, 4096, 1.5e-7),
                                            (1160, 6933, 1.4e-7), (2048, 8192, 1.7e-7)])
def test_batched_factor_is_as_accurate_as_float32_multiply_adds(K, tokens, limit):
    H, ref = _spd_factor64(K, tokens)
    Hs = [H.clone() for _ in range(3)]
    ops.gptq_factor_batched(Hs)
    for U in Hs:
        assert float((U.double() - ref).norm() / ref.norm()) <= limit


# the last column after all the corrections: the earlier rows of U times 2^20 keep their errors out of the loss, every
# code is zero (a huge scale), so the loss is half the square of that column's error.  `limit` as above, relative to the
# column's root mean square
@pytest.mark.parametrize("N,K,tokens,limit", [(1001, 520, 1500, 2.8e-7), (6000, 520, 1500, 3.2e-7),
                                              (1001, 2048, 8192, 4.0e-7)])
def test_batched_sweep_is_as_accurate_as_float32_multiply_adds(N, K, tokens, limit):
    _, ref = _spd_factor64(K, tokens)
    U = ref.float().contiguous()
    U[:-1] *= 2.0 ** 20
    w = (torch.randn(N, K, generator=torch.Generator(device=DEV).manual_seed(N), device=DEV) * 0.02).bfloat16()
    last = torch.linalg.solve_triangular(U.double(), w.double(), upper=True, left=False)[:, -1].abs()
    args = args_from(SCHEMES["W8_CHANNEL"])
    scale = torch.full((N, 1), 1e4, device=DEV).bfloat16()
    losses = ops.gptq_sweep_batched([w.float() for _ in range(3)], [U] * 3, [scale] * 3, None, args)
    for row in losses:
        error = (2.0 * row.double()).sqrt() - last
        assert float(error.pow(2).mean().sqrt() / last.pow(2).mean().sqrt()) <= limit


# every code zero: the errors of a row are W U^-1, their sum of squares the loss.  `limit`: the same error (relative, root
# mean square over the rows) with sums of 128 terms
@pytest.mark.parametrize("N,K,tokens,limit", [(1001, 520, 1500, 2.3e-7), (1001, 1160, 6933, 1.6e-7), (6000, 1160, 6933, 1.6e-7)])
def test_sweep_losses_are_summed_in_short_runs(N, K, tokens, limit):
    _, ref = _spd_factor64(K, tokens)
    U = ref.float().contiguous()
    w = (torch.randn(N, K, generator=torch.Generator(device=DEV).manual_seed(N), device=DEV) * 0.02).bfloat16()
    errors = torch.linalg.solve_triangular(U.double(), w.double(), upper=True, left=False)
    total = 0.5 * (errors * errors).sum(1)
    scale = torch.full((N, 1), 1e4, device=DEV).bfloat16()
    losses = ops.gptq_sweep(w.float(), U, scale, None, args_from(SCHEMES["W8_CHANNEL"]))
    assert float(((losses.double() - total) / total).pow(2).mean().sqrt()) <= limit


def test_status_of_a_deferred_sweep_does_not_keep_its_workspace():
    args = args_from(SCHEMES["W4A16"])
    problems = [_problem(64, 640, seed=i) for i in range(2)]
    mods = [_lin(w, args) for w, _ in problems]
    factors = gptq.factor_hessians_batched([H.clone().to(DEV) for _, H in problems], 0.01, None)
    words = [gptq.quantize_weights_batched(mods, args, factors)[0][1]["_status"]]
    words.append(gptq.quantize_weight(mods[0], args, None, factor=factors[0], defer=True)[1]["_status"])
    for w in words:
        assert int(w) == 0 and w.untyped_storage().nbytes() == 4


@pytest.mark.parametrize("scheme", ["FP8_DYNAMIC", "W4A16_ASYM"])
def test_parameters_of_a_batch_own_their_storage(scheme):
    """Saving or dropping one expert must not take the others' parameters along; values as a module by itself gets them."""
    K, N, count = 256, 64, 16
    parent = torch.nn.Module()
    for k in range(count):
        lin = torch.nn.Linear(K, N, bias=False, device=DEV, dtype=torch.bfloat16)
        lin.weight.data = synth_weight(N, K, k).to(DEV)
        parent.add_module(f"expert_{k}", lin)
    mod = GPTQModifier(targets="Linear", scheme=scheme, actorder=None)
    mod.on_initialize(parent)
    mod.on_calibration_start(parent)
    x = synth_acts(2, 512, K, 0).to(DEV)
    expected = []
    for lin in parent.children():
        args = lin.quantization_scheme.weights
        expected.append(ops.qparams(*ops.observe_minmax(lin.weight.data, args), args))
        mod.calibrate_module(lin, (x,), None)
    mod.on_sequential_epoch_end(parent, list(parent.modules()))
    for lin, (scale, zp) in zip(parent.children(), expected):
        assert lin.quantization_status == "frozen"
        for p in lin.parameters():
            assert p.untyped_storage().nbytes() == p.numel() * p.element_size()
        assert bits_equal(lin.weight_scale, scale) and bits_equal(lin.weight_zero_point, zp)


def test_entry_points_without_workspace():
    """b200q_gptq_factor_batched and b200q_gptq_sweep_batched give what the calls with a workspace give."""
    lib, args, K, N, count = _lib.load(), args_from(SCHEMES["W4A16"]), 640, 96, 3
    Hs = [_spd(K, i).to(DEV) for i in range(count)]
    many, batched = [H.clone() for H in Hs], [H.clone() for H in Hs]
    ops.gptq_factor_batched(many)
    scratch = [torch.empty(lib.b200q_gptq_factor_batched_workspace_bytes(K, 1) // 4, device=DEV) for _ in range(count)]
    status = torch.full((count, 4), 7, dtype=torch.int32, device=DEV)
    table = ops._pointer_table([batched, scratch])
    _lib.check(lib.b200q_gptq_factor_batched(table[0].data_ptr(), table[1].data_ptr(), count, K, K, status.data_ptr(),
                                             _lib.stream_ptr()), "factor")
    assert int(status.abs().max()) == 0 and all(bits_equal(a, b) for a, b in zip(many, batched))
    ws = [synth_weight(N, K, seed=i).to(DEV) for i in range(count)]
    scales = [ops.qparams(*ops.observe_minmax(w, args), args)[0] for w in ws]
    a, b = [w.float() for w in ws], [w.float() for w in ws]
    losses = ops.gptq_sweep_batched(a, many, scales, None, args)
    got = torch.empty_like(losses)
    table = ops._pointer_table([b, many, scales, got])
    _lib.check(lib.b200q_gptq_sweep_batched(table[0].data_ptr(), table[1].data_ptr(), table[2].data_ptr(), _lib.BF16, None,
                                            None, None, table[3].data_ptr(), count, N, K, K, K, args.c_struct(), 128,
                                            _lib.stream_ptr()), "sweep")
    assert bits_equal(got, losses) and all(bits_equal(x, y) for x, y in zip(a, b))
    assert lib.b200q_take_wait_status() == 0


def test_noted_status_word_is_reported_once():
    lib = _lib.load()
    for word, expected in ((0, 0), (-4, -4)):
        _lib.check(lib.b200q_note_wait_status(torch.full((1,), word, dtype=torch.int32, device=DEV).data_ptr(),
                                              _lib.stream_ptr()), "note")
        assert lib.b200q_take_wait_status() == expected and lib.b200q_take_wait_status() == 0


# one problem: `limit` is the error of the same solve with rank-128 tensor-core updates and float32 multiply-adds inside a block
@pytest.mark.parametrize("K,tokens,limit", [(256, 600, 7.3e-7), (768, 4096, 4.3e-7), (2048, 8192, 6.0e-7), (4096, 9000, 1.28e-6)])
def test_factor_is_as_accurate_as_rank_128_updates(K, tokens, limit):
    H, ref = _spd_factor64(K, tokens)
    assert ops.gptq_factor(H) == 0
    assert float((H.double() - ref).norm() / ref.norm()) <= limit


@pytest.mark.parametrize("N,K,tokens,limit", [(1001, 256, 600, 3.7e-7), (1001, 520, 1500, 9.2e-7), (6000, 1160, 6933, 4.8e-7),
                                              (1001, 4096, 9000, 7.0e-7)])
def test_sweep_is_as_accurate_as_rank_128_updates(N, K, tokens, limit):
    _, ref = _spd_factor64(K, tokens)
    U = ref.float().contiguous()
    U[:-1] *= 2.0 ** 20
    w = (torch.randn(N, K, generator=torch.Generator(device=DEV).manual_seed(N), device=DEV) * 0.02).bfloat16()
    last = torch.linalg.solve_triangular(U.double(), w.double(), upper=True, left=False)[:, -1].abs()
    scale = torch.full((N, 1), 1e4, device=DEV).bfloat16()
    losses = ops.gptq_sweep(w.float(), U, scale, None, args_from(SCHEMES["W8_CHANNEL"]))
    error = (2.0 * losses.double()).sqrt() - last
    assert float(error.pow(2).mean().sqrt() / last.pow(2).mean().sqrt()) <= limit


# every code zero and the last column alone in the loss, as above, with columns of activations 2^-18 .. 2^18 in size: even
# weights; weights that go the other way, so that all columns' errors count alike; even weights and every second column tiny
# and without correlation to the others, so that only the smallest errors reach the last column.  Three times the limit of
# equal sizes: either side of a product spans 2^18, and of its smallest values 21 to 22 bits are kept
@pytest.mark.parametrize("N,K,tokens", [(1001, 520, 1500), (1001, 1160, 6933), (6000, 520, 1500)])
@pytest.mark.parametrize("grading", ["activations", "weights", "groups"])
def test_sweep_of_columns_graded_in_size(grading, N, K, tokens):
    H, ref = _spd_factor64(K, tokens)
    e = torch.randint(-18, 19, (K,), generator=torch.Generator().manual_seed(K)).to(DEV)
    w = (torch.randn(N, K, generator=torch.Generator(device=DEV).manual_seed(N), device=DEV) * 0.02).bfloat16().float()
    if grading == "groups":
        odd = torch.arange(K, device=DEV) % 2 == (K - 1) % 2
        e = torch.where(odd, -18, 18)
        H = torch.where(odd[:, None] == odd[None, :], H, 0.0).double()
        L = torch.linalg.cholesky(H.flip(0, 1))
        ref = torch.linalg.solve_triangular(L, torch.eye(K, device=DEV, dtype=torch.float64), upper=False).flip(0, 1)
    U = torch.ldexp(ref, -e).float().contiguous()   # H = S R S has U S^-1
    if grading == "weights":
        w = torch.ldexp(w, -e)
    U[:-1] *= 2.0 ** 60
    last = torch.linalg.solve_triangular(U.double(), w.double(), upper=True, left=False)[:, -1].abs()
    scale = torch.full((N, 1), 2.0 ** 40, device=DEV).bfloat16()
    losses = ops.gptq_sweep(w.clone(), U, scale, None, args_from(SCHEMES["W8_CHANNEL"]))
    error = (2.0 * losses.double()).sqrt() - last
    assert float(error.pow(2).mean().sqrt() / last.pow(2).mean().sqrt()) <= 3 * (9.2e-7 if K == 520 else 4.8e-7)
