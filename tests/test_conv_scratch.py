"""The scratch of decode_conv for the activated rows: a CUDA graph holds its address for as long as it is replayed, so a buffer that
was handed out once stays the state's, whatever larger calls follow."""
import gc

import pytest
import torch

from leapquant_b200.state import LeapQuantState

K = V = 128


def rows_handed_out(st, sizes):
    """Address and rows of the scratch that each of a series of calls passes on, with the kernels left out."""
    out = []
    st._kconv = lambda x, cs, w, b, i, mixed: out.append((mixed.data_ptr(), tuple(mixed.shape)))
    st.decode = lambda *a: None
    for n in sizes:
        st.decode_conv(None, torch.empty(n, 4), None, None, None, None, None, None, None, torch.zeros(n, dtype=torch.int32), None)
    return out


def owned(st):
    found = {}
    for v in vars(st).values():
        for t in v if isinstance(v, (list, tuple)) else [v]:
            if isinstance(t, torch.Tensor):
                found[t.data_ptr()] = t
    return found


@pytest.mark.parametrize("sizes", [(40, 100, 40), (1, 65, 64, 700, 3), tuple(range(1, 300))])
def test_scratch_stays_owned(sizes):
    st = LeapQuantState.__new__(LeapQuantState)
    st.conv_one_launch, st._mixed, st.H, st.K, st.HV, st.V, st.NS = False, None, 1, K, 2, V, 900
    for name in ("_mixed_old",):
        st.__dict__.setdefault(name, [])
    got = rows_handed_out(st, sizes)
    gc.collect()
    mine = owned(st)
    for (ptr, shape), n in zip(got, sizes):
        assert shape == (n, 2 * K + 2 * V)
        assert ptr in mine and mine[ptr].shape[0] >= n, "a buffer that a graph may hold went back to the allocator"
    assert sum(t.shape[0] for t in mine.values()) <= 4 * max(max(sizes), 32)


@pytest.mark.gpu
def test_graph_replay_after_a_larger_call():
    """Eager call, capture, eager call with more rows, other tensors in the freed memory, replay: the replay computes what the capture
    would have, and leaves those tensors alone."""
    H, HV, NS, L = 2, 4, 140, 16
    C = 2 * H * K + HV * V

    def run(larger):
        g = torch.Generator().manual_seed(3)
        r = lambda *s: torch.randn(*s, generator=g).to(torch.bfloat16).cuda()
        ssm = (0.1 * torch.randn(NS, HV, V, K, generator=g)).cuda()
        st = LeapQuantState(ssm, H, L=L)
        st.quantize(ssm, torch.arange(1, NS, dtype=torch.int32, device="cuda"))
        conv, w = r(NS, 3, C).transpose(1, 2), r(C, 4)
        x, a, b = r(128, C), r(128, HV), r(128, HV)
        A_log, dtb = torch.rand(HV, generator=g).cuda(), torch.rand(HV, generator=g).cuda()
        idx = torch.arange(1, 129, dtype=torch.int32, device="cuda")
        out = torch.zeros(128, HV, V, dtype=torch.bfloat16, device="cuda")
        call = lambda n, i: st.decode_conv(ssm, x[:n], conv, w, None, a[:n], b[:n], A_log, dtb, i[:n], out[:n])
        null = torch.zeros_like(idx)
        call(32, null)                                             # (padding rows only: allocates, changes no state)
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            call(32, idx)
        others = []
        if larger:
            call(128, null)
            torch.cuda.synchronize()
            others = [torch.full((64, C), 7.0, dtype=torch.bfloat16, device="cuda") for _ in range(8)]
        graph.replay()
        torch.cuda.synchronize()
        assert all(bool((t == 7.0).all()) for t in others)
        return out[:32].clone(), st.Kbuf.clone(), st.Ubuf.clone()

    for p, q in zip(run(False), run(True)):
        assert torch.equal(p, q)
