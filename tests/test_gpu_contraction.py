"""The error of the F16 contraction that the proofs of irc_cert.cu bound: operand
rows as irc_tc_host.cu lays them out, multiplied on the tensor cores with FP32
accumulation, against the distances of the same rounded rows in FP64.  The proof
charges 2^-15 (|x|^2 + |y|^2 + tau) + 1e-6; 70 truncating FP32 additions of terms
that sum to twice that are below 2^-16 of it, which is what is asked for here."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def split3(v):
    h = v.half()
    m = (v - h.float()).half()
    return h, m, (v - h.float() - m.float()).half()


@pytest.mark.parametrize("d", [1, 9, 24, 33, 45, 55])
@pytest.mark.parametrize("norm", [0.05, 1.0, 15.0, 64.0, 240.0])
def test_contraction_error(gpu, d, norm):
    g = torch.Generator(device=gpu).manual_seed(d)
    n = 2048
    c = torch.randn(20, d, device=gpu, generator=g)
    x = c[torch.randint(0, 20, (n,), device=gpu, generator=g)] + 0.1 * torch.randn(n, d, device=gpu, generator=g)
    x = x / (x * x).sum(1).max().sqrt() * norm                 # the longest row has this norm
    X = x.half()
    na = torch.zeros(n, device=gpu)
    for k in range(d):
        na = torch.addcmul(na, X[:, k].float(), X[:, k].float())
    tau = na.mean() * 0.01
    Q = torch.zeros(n, 64, device=gpu, dtype=torch.half)
    C = torch.zeros_like(Q)
    Q[:, :d], C[:, :d] = -2 * X, X
    for i, p in enumerate(split3(na)):
        Q[:, d + i], C[:, d + i], Q[:, d + 3 + i], C[:, d + 3 + i] = p, 1, 1, p
    for i, p in enumerate(split3(-tau)):
        Q[:, d + 6 + i], C[:, d + 6 + i] = p, 1
    V = torch.mm(Q, C.t(), out_dtype=torch.float32).double()
    Y = X.double()
    N = (Y * Y).sum(1)
    D = ((Y[:, None] - Y[None]) ** 2).sum(2) - tau.double()
    err = (V - D).abs() - 1e-6
    assert bool((err <= 2.0 ** -16 * (N[:, None] + N[None] + tau.double())).all())
