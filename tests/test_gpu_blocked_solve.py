"""The blocked form of a factor and the sweep that takes it, against float64: edges of squares, of CTAs and of the range."""
import pytest
import torch

from helpers import args_from
from llm_compressor_b200 import ops
from llm_compressor_b200.quant_args import QuantizationArgs
from test_gpu_batched_solve import SCHEMES, _spd_factor64
from test_gpu_variants import _spd

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _blocks64(H):
    """float64: (U, blocked form) of H"""
    K = H.shape[0]
    V = torch.linalg.cholesky(H.flip(0, 1)).flip(0, 1)
    U = torch.linalg.solve_triangular(V, torch.eye(K, device=H.device, dtype=H.dtype), upper=True)
    F = U.clone()
    for c in range(512, K, 512):
        F[:c, c:c + 512] = -V[:c, c:c + 512] @ U[c:c + 512, c:c + 512]
    return U, F


def _rows(w, half):
    """w as the kept columns are: bf16 or float32, rows of 16-byte pieces"""
    N, K = w.shape
    kept = torch.full((N, (K + 7) // 8 * 8), float("nan"), device=DEV, dtype=torch.bfloat16 if half else torch.float32)[:, :K]
    kept.copy_(w)
    return kept


# a square and a column, remainders that are and are not multiples of 4 and 32, whole squares, three of them and a part
@pytest.mark.parametrize("K", [513, 520, 640, 1030, 1160, 1536, 2500])
def test_blocked_factor_at_block_edges(K):
    H = _spd(K, K)
    ref = _blocks64(H.float().double())[1]
    got = H.float()
    assert int(ops.gptq_factor_async(got, blocks=True).abs().max()) == 0
    # float32 with products of 22 bits and short runs: U itself is held to 5e-6 at this conditioning
    assert float((got.triu().double() - ref).norm() / ref.norm()) < 5e-6
    bad = H.float()
    bad[3, 3] = -1.0
    assert ops.gptq_factor_async(bad, blocks=True).tolist()[0:2] == [1, K - 3]


# rows: one, part of a CTA, few (far columns beside the next sweep), the most that one CTA an SM carries
@pytest.mark.parametrize("N,K", [(1, 513), (33, 520), (64, 1160), (97, 2100), (2400, 1030), (4736, 1537)])
@pytest.mark.parametrize("scheme", ["W8_CHANNEL", "W4_ASYM"])
def test_blocked_sweep_at_edges_of_blocks(N, K, scheme):
    assert ops.gptq_sweep_takes_blocks(N, K)
    U, F = _blocks64(_spd(K, K))
    g = torch.Generator(device=DEV).manual_seed(N)
    w = (torch.randn(N, K, generator=g, device=DEV) * 0.02).bfloat16().double()
    asym = scheme == "W4_ASYM"
    scale = torch.full((N, 1), 0.01 if asym else 5e-4, device=DEV).bfloat16()
    zp = (torch.arange(N, device=DEV) % 5 - 2).to(torch.int8).view(N, 1) if asym else None
    args = QuantizationArgs(num_bits=4 if asym else 8, type="int", symmetric=not asym, strategy="channel")
    lo, hi = (-8, 7) if asym else (-128, 127)
    x, s = w.clone(), scale.double()
    z = zp.double() if asym else torch.zeros(N, 1, dtype=torch.float64, device=DEV)
    q, loss = torch.zeros_like(w), torch.zeros(N, dtype=torch.float64, device=DEV)
    close = torch.zeros(N, dtype=torch.bool, device=DEV)
    for i in range(K):
        c = (x[:, i:i + 1] / s + z).clamp(lo, hi)
        # float32 sums (errors below 1e-6 of the weights' size, 3e-5 of a step) may turn a code this close to a boundary
        close |= ((c - c.floor() - 0.5).abs() < 1e-4)[:, 0]
        q[:, i] = ((c.round() - z) * s).bfloat16().double()[:, 0]
        e = (x[:, i] - q[:, i]) / U[i, i]
        loss += e * e / 2
        x[:, i + 1:] -= e[:, None] * U[i, i + 1:]
    W = w.float()
    losses, status = ops.gptq_sweep(W, F.float().contiguous(), scale, zp, args, return_status=True, original=_rows(w, asym))
    assert int(status) == 0
    sure = ~close
    assert torch.equal(W.double()[sure], q[sure])
    assert torch.allclose(losses.double()[sure], loss[sure], rtol=1e-4)
    assert float((W.double() != q).double().mean()) < 0.05


# every code zero, the last column alone in the loss (rows of U times 2^20 keep the others out); columns of equal sizes and
# 2^-14 .. 2^14, with even weights and with weights that go the other way.  Limits: of the sweep that takes U
@pytest.mark.parametrize("N,K,tokens,limit", [(1001, 520, 1500, 9.2e-7), (1001, 1160, 6933, 4.8e-7), (1001, 4096, 9000, 7.0e-7)])
@pytest.mark.parametrize("grading", ["none", "activations", "weights"])
def test_blocked_sweep_is_as_accurate_as_with_the_factor(grading, N, K, tokens, limit):
    H, _ = _spd_factor64(K, tokens)
    e = torch.randint(-14, 15, (K,), generator=torch.Generator().manual_seed(K)).to(DEV)
    if grading == "none":
        e = torch.zeros_like(e)
    H = torch.ldexp(torch.ldexp(H.double(), e), e[:, None])
    U, F = _blocks64(H)
    w = (torch.randn(N, K, generator=torch.Generator(device=DEV).manual_seed(N), device=DEV) * 0.02).bfloat16().float()
    if grading == "weights":
        w = torch.ldexp(w, -e)
    last = torch.linalg.solve_triangular(U, w.double(), upper=True, left=False)[:, -1].abs()
    F = F.float().contiguous()
    for c in range(0, K, 512):
        F[c:c + 512, c:c + 512] *= 2.0 ** 50
    F[-1] *= 2.0 ** -50
    scale = torch.full((N, 1), 2.0 ** 40, device=DEV).bfloat16()
    losses = ops.gptq_sweep(w.clone(), F, scale, None, args_from(SCHEMES["W8_CHANNEL"]), original=_rows(w, False))
    error = (2.0 * losses.double()).sqrt() - last
    measured = float(error.pow(2).mean().sqrt() / last.pow(2).mean().sqrt())
    print(grading, K, measured)
    assert measured <= limit * (1 if grading == "none" else 3)
