"""What lq_quantize stores is fixed to the last bit: an engine that quantizes a state, dequantizes it and quantizes it again feeds a
rounding of the first pass into codes of the second, so two builds that add in different orders drift apart.

  factors   those of lq_lowrank on the transposed state, rounded to f16: sums of 64 + 64 products in index order, modified
            Gram-Schmidt by pairs (the two kernels share no code but that order)
  scales    Sk = sqrt of the column means of |E| (64 + 64 rows in order), Sv = the largest true quotient |E / Sk| of a row
  codes     rint(E / (Sk Sv) * 127) with true divisions
"""
import numpy as np
import pytest
import torch

from oracle import lq_oracle as O
from test_gpu_quantize import KINDS, state

K = V = 128


def restated(S, U, Q):
    """Sk, Sv, codes of fp32 states S [n, V, K] given the stored factors U [n, R, K], Q [n, R, V]: fp32 operations one by one (a fused
    multiply-add as one rounding of its value in 64 bits, which holds the product of two f16 values exactly)."""
    E = S.float()
    for r in range(U.shape[1]):
        E = (E.double() - Q[:, r, :, None].double() * U[:, r, None, :].double()).float()
    A = E.abs()
    halves = []
    for lo in (0, 64):
        acc = torch.zeros_like(A[:, 0])
        for row in range(lo, lo + 64):
            acc = acc + A[:, row]
        halves.append(acc)
    Sk = torch.from_numpy(np.sqrt(((halves[0] + halves[1]) / 128).numpy())).clamp_min(1e-12)     # (torch's fp32 root is not rounded to nearest)
    Sv = (E / Sk[:, None, :]).abs().amax(-1).clamp_min(1e-12)
    codes = torch.round((E / (Sk[:, None, :] * Sv[:, :, None])).double() * 127).to(torch.int8)
    return Sk, Sv, codes


def quantized(S, R, iters):
    """Codes, scales and factors of the heads S [NS, HV, V, K], slot 0 left out, on the CPU and flat over the heads."""
    from leapquant_b200.kernels import make_quantize
    from leapquant_b200.state import state_views
    NS, HV = S.shape[:2]
    ssm = S.cuda()
    v = state_views(ssm, R)
    z = lambda *s, **kw: torch.zeros(*s, device="cuda", **kw)
    make_quantize(NS, HV, K, V, 16, ssm.stride(0), R=R, ITERS=iters)(
        ssm, v["Sq"], v["Sk"], v["Sv"], v["uq"], z(NS, HV, 16), z(NS, HV, 1), z(NS, HV, dtype=torch.int32), O.make_q0(V, R).cuda(),
        torch.arange(1, NS, dtype=torch.int32, device="cuda"), None)
    return {n: v[n][1:].cpu().flatten(0, 1) for n in ("Sq", "Sk", "Sv", "uq")}


def heads(R, iters, HV=29):
    """States of every kind, 551 heads: more than the kernel holds at once."""
    g = torch.Generator().manual_seed(100 * R + iters)
    kinds = [k for k in KINDS if k != "huge"] + ["noise", "low rank"] * 6
    S = torch.zeros(len(kinds) + 1, HV, V, K)
    for i, kind in enumerate(kinds):
        S[i + 1] = state(kind, HV, g).float()
    return S, [k for k in kinds for _ in range(HV)]


def same(name, got, want, kinds):
    at = (got != want).nonzero().tolist()
    assert not at, (name, len(at), [(kinds[i[0]], i, float(got[tuple(i)]), float(want[tuple(i)])) for i in at[:4]])


CASES = pytest.mark.parametrize("R,iters", [(4, 1), (4, 0), (4, 2), (8, 3), (8, 1)])


@pytest.mark.gpu
@CASES
def test_factor_bits(R, iters):
    from leapquant_b200.kernels import lowrank_factor
    S, kinds = heads(R, iters)
    got = quantized(S, R, iters)
    U, Q = lowrank_factor(S.transpose(-1, -2).contiguous().cuda(), R, iters)      # [NS, HV, K, R], [NS, HV, V, R]
    want = torch.cat([U, Q], -2).transpose(-1, -2).to(torch.float16)[1:].cpu().flatten(0, 1)
    same("uq", got["uq"], want, kinds)
    # column scales: the same order of sums
    Sk = restated(S[1:].flatten(0, 1), want[..., :K], want[..., K:])[0]
    same("Sk", got["Sk"], Sk, kinds)


@pytest.mark.gpu
@CASES
def test_scale_and_code_bits(R, iters):
    S, kinds = heads(R, iters)
    got = quantized(S, R, iters)
    _, Sv, codes = restated(S[1:].flatten(0, 1), got["uq"][..., :K], got["uq"][..., K:])
    same("Sv", got["Sv"], Sv, kinds)
    same("Sq", got["Sq"], codes, kinds)


@pytest.mark.gpu
@pytest.mark.parametrize("R,iters", [(4, 1), (8, 3)])
def test_orthogonality_and_energy(R, iters):
    """Of the stored value factors, on states whose columns P are nearly dependent (one direction 1e5 times the rest) and others:
    |Q^T Q - I| <= 2^-9 (f16 values: 2^-11 of each of two unit columns) + 16 eps cond (modified Gram-Schmidt loses eps cond), and
    the part they leave is that of the 64-bit iteration to the spacing of the factors."""
    S, kinds = heads(R, iters, HV=3)
    got = quantized(S, R, iters)
    U, Q = got["uq"][..., :K].double(), got["uq"][..., K:].double()
    Q0 = O.make_q0(V, R).double()
    for i, kind in enumerate(kinds):
        if kind not in ("noise", "low rank", "steep", "parallel"):
            continue
        A = S[1:].flatten(0, 1)[i].double()
        X, cond = Q0, 1.0
        for _ in range(iters):
            P = A.T @ X
            cond = max(cond, float(torch.linalg.cond(P)))
            X = A @ torch.linalg.qr(P)[0]
            cond = max(cond, float(torch.linalg.cond(X)))
            X = torch.linalg.qr(X)[0]
        off = float((Q[i] @ Q[i].T - torch.eye(R, dtype=torch.float64)).abs().max())
        assert off <= 2 ** -9 + 16 * 2 ** -24 * cond, (kind, off, cond)
        left, best = (A - Q[i].T @ U[i]).norm(), (A - X @ (X.T @ A)).norm()
        assert float(left) <= float(best) + (2 ** -10 + 16 * 2 ** -24 * cond) * float(A.norm()), (kind, float(left), float(best), cond)


@pytest.mark.gpu
def test_kda_window_reset():
    """quantize of a KDA state resets the listed windows (weights 0, decay 0, gates 1, count 0) and no other."""
    from leapquant_b200.state import LeapQuantState
    NS, HV, L = 9, 3, 24
    ssm = (0.1 * torch.randn(NS, HV, V, K, generator=torch.Generator().manual_seed(1))).cuda()
    st = LeapQuantState(ssm, HV, kda=True, L=L, R=8)
    for t, x in ((st.Wbuf, 0.5), (st.Pbuf, -0.25), (st.Gbuf, 0.75), (st.hcnt, 5)):
        t.fill_(x)
    st.quantize(ssm, torch.tensor([2, 0, 7, -1, 4, NS], dtype=torch.int32, device="cuda"))
    mine = torch.tensor([2, 7, 4], device="cuda")
    rest = torch.tensor([0, 1, 3, 5, 6, 8], device="cuda")
    for t, new, old in ((st.Wbuf, 0.0, 0.5), (st.Pbuf, 0.0, -0.25), (st.Gbuf, 1.0, 0.75), (st.hcnt, 0, 5)):
        assert bool((t[mine] == new).all()) and bool((t[rest] == old).all())


@pytest.mark.gpu
@pytest.mark.parametrize("R,iters", [(4, 1), (8, 3)])
def test_not_a_number_stays_in_its_head(R, iters):
    from leapquant_b200 import _lib
    S, _ = heads(R, iters, HV=2)
    clean = quantized(S, R, iters)
    bad = [3, 8, 21]
    flat = S[1:].flatten(0, 1)
    for n, x in zip(bad, (float("nan"), float("inf"), -float("inf"))):
        flat[n, 17, 5] = x
    S[1:] = flat.view_as(S[1:])
    got = quantized(S, R, iters)
    rest = [n for n in range(flat.shape[0]) if n not in bad]
    for name in clean:
        assert torch.equal(got[name][rest].view(torch.int8), clean[name][rest].view(torch.int8)), name
    assert _lib.device_status() == 0
