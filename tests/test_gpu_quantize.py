"""lq_quantize over more heads than its CTAs hold at once, with padding rows between them, on states of every rank: the stored
checkpoint stands for the state to half a code, the factors are those of the 64-bit subspace iteration."""
import pytest
import torch

from oracle import lq_oracle as O

K = V = 128
KINDS = ("noise", "low rank", "zero", "one token", "two tokens", "steep", "parallel", "huge")


def state(kind, HV, g):
    r = lambda *s: torch.randn(*s, generator=g, dtype=torch.float64)
    if kind == "zero":
        return torch.zeros(HV, V, K, dtype=torch.float64)
    if kind in ("one token", "two tokens"):                       # fewer tokens than compensator tokens: rank deficient
        n = 1 if kind == "one token" else 2
        return r(HV, V, n) @ r(HV, n, K)
    if kind in ("steep", "parallel"):                             # singular values over six decades; one direction 1e5 times the rest
        u, v = torch.linalg.qr(r(HV, V, V))[0], torch.linalg.qr(r(HV, K, K))[0]
        s = 10.0 ** torch.linspace(0, -6, K, dtype=torch.float64) if kind == "steep" else torch.cat(
            [torch.ones(1, dtype=torch.float64), torch.full((K - 1,), 1e-5, dtype=torch.float64)])
        return (u * s) @ v
    S = 0.1 * r(HV, V, K)
    if kind == "low rank":
        S += r(HV, V, 4) @ r(HV, 4, K)
    return S * (1e19 if kind == "huge" else 1.0)


@pytest.mark.gpu
@pytest.mark.parametrize("rows,HV,R,kda", [(1, 1, 4, False), (9, 16, 4, False), (230, 3, 4, False), (150, 4, 8, True), (8, 5, 8, False)])
def test_quantize_many_heads(rows, HV, R, kda):
    from leapquant_b200.state import LeapQuantState
    g = torch.Generator().manual_seed(rows)
    NS = rows + 2
    kinds = [KINDS[i % len(KINDS)] for i in range(rows)]
    if rows > 16:                                                  # (the rank-deficient kinds once, the rest well conditioned)
        kinds = list(KINDS) + ["noise" if i % 2 else "low rank" for i in range(rows - len(KINDS))]
    S64 = torch.zeros(NS, HV, V, K, dtype=torch.float64)
    slots = torch.randperm(NS - 1, generator=g)[:rows] + 1
    for s, kind in zip(slots.tolist(), kinds):
        S64[s] = state(kind, HV, g)
    S = S64.float()
    ssm = S.cuda()
    st = LeapQuantState(ssm, HV, kda=kda, L=16, R=R)
    for t, v in ((st.Wbuf, 0.5), (st.Pbuf, 0.25), (st.hcnt, 3)):
        t.fill_(v)
    idx = torch.zeros(2 * rows + 1, dtype=torch.int32)             # every other row is padding: null, negative or past the last slot
    idx[1::2] = slots.to(torch.int32)
    idx[2::6] = -1
    idx[4::6] = NS
    st.quantize(ssm, idx.cuda())
    torch.cuda.synchronize()
    v = {n: t.double().cpu() for n, t in st.views(ssm).items() if n in ("Sq", "Sk", "Sv", "uq")}
    U, Q = v["uq"][slots][..., :K], v["uq"][slots][..., K:]
    QU = Q.transpose(-1, -2) @ U
    step = v["Sk"][slots][:, :, None, :] * v["Sv"][slots][:, :, :, None] / 127
    want = S[slots].double()
    # half a code, and a few fp32 roundings of the magnitudes that cancel in the residual
    slack = 0.502 * step + 6e-7 * (want.abs() + Q.abs().transpose(-1, -2) @ U.abs())
    err = (v["Sq"][slots] * step + QU - want).abs()
    assert bool((err <= slack).all()), [k for k, e in zip(kinds, (err > slack).flatten(1).any(1)) if e]
    assert int(st.hcnt[slots.cuda()].abs().max()) == 0 and float(st.Wbuf[slots.cuda()].abs().max()) == 0
    assert float((st.Pbuf[slots.cuda()] - (0.0 if kda else 1.0)).abs().max()) == 0
    rest = torch.tensor([s for s in range(NS) if s not in set(slots.tolist())])
    assert torch.equal(ssm[rest.cuda()].cpu(), S[rest]) and int(st.hcnt[rest.cuda()].min()) == 3
    # well-conditioned states: the rank-R part of the 64-bit iteration, to the spacing of the f16 factors
    Q0 = O.make_q0(V, R).double()
    for i, kind in enumerate(kinds):
        if kind not in ("noise", "low rank"):
            continue
        X, A = Q0.expand(HV, V, R), want[i]
        for _ in range(3 if kda else 1):
            P = torch.linalg.qr(A.transpose(-1, -2) @ X)[0]
            X = torch.linalg.qr(A @ P)[0]
        ref = X @ (X.transpose(-1, -2) @ A)
        rel = float((QU[i] - ref).norm() / ref.norm())
        assert rel < 1e-3, (kind, rel)                             # (f16 factors: 2 * 2^-12 of each product)
