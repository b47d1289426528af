"""The walk of an mLSTM's matrix memory in chunks on the tensor cores against the recurrence in float64, beside the scan in
float32 products that it stands in for."""

import types

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _recurrence(q, k, v, a, b, S, n):
    """All float64, one head: q, k [t, dk], v [t, dv], a, b [t]; returns [t, dv + 1] and the state after the last token."""
    out = []
    for t in range(q.shape[0]):
        S = a[t] * S + b[t] * torch.outer(k[t], v[t])
        n = a[t] * n + b[t] * k[t]
        out.append(torch.cat([S.T @ q[t], (n @ q[t])[None]]))
    return torch.stack(out), S, n


@pytest.mark.parametrize("heads,dk,dv,lens,forget", [(2, 128, 128, [130, 64, 1], 2.0), (3, 16, 32, [65, 33, 200], 0.0), (1, 64, 16, [300], -4.0),
                                                     (1, 256, 48, [100, 63], 6.0)])
def test_mlstm_chunked(heads, dk, dv, lens, forget):
    from bare_cuda_4gib_b200.kernels import lib as K, linear_attention as LA, mlstm as MK
    torch.manual_seed(dk + dv)
    rows, slots, dvp, cap = sum(lens), len(lens) + 2, dv + 4, 15.0
    ints = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    ctx = types.SimpleNamespace(seq_slot=ints([i + 1 for i in range(len(lens))]), seq_q_start=ints([sum(lens[:i]) for i in range(len(lens))]),
                                seq_q_len=ints(lens), n_seqs=len(lens), n_tokens=rows, max_q_len=max(lens), stream=K.stream_handle(),
                                dtype=torch.float32)
    kd, vd = heads * dk, heads * dv
    u = torch.randn(rows, 2 * kd + 2 * vd, device=DEV).to(torch.bfloat16)
    z = torch.randn(rows, 2 * heads, device=DEV)
    bias = [torch.randn(heads, device=DEV), forget + torch.randn(heads, device=DEV)]
    m0 = torch.randn(slots, heads, device=DEV)
    coef = torch.empty(rows, heads * 4, device=DEV)
    la, b = torch.empty(rows, heads, device=DEV), torch.empty(rows, heads, device=DEV)
    MK.gates(ctx, z, 0, heads, bias[0], bias[1], cap, m0.clone(), coef, heads, la, b)
    assert torch.equal(coef.view(rows, heads, 4)[..., 1], b) and torch.allclose(coef.view(rows, heads, 4)[..., 0], la.exp(), rtol=1e-6, atol=0)
    start = torch.randn(slots, heads, dk, dvp, device=DEV)
    start[..., dv + 1:] = 0.0
    state, out = start.clone(), torch.full((rows, heads * dvp), float("nan"), device=DEV)
    MK.chunked(ctx, u, 0, kd, 2 * kd, la, b, state, out, heads, dk, dv, dk ** -0.5)
    # the scan, in float32
    qf, kf, vf = torch.empty(rows, kd, device=DEV), torch.empty(rows, kd, device=DEV), torch.empty(rows, heads * dvp, device=DEV)
    decay, scanned, walked = torch.empty(rows, heads, device=DEV), torch.empty(rows, heads * dvp, device=DEV), start.clone()
    MK.operands(ctx, u, 0, kd, 2 * kd, coef, qf, kf, decay, vf, heads, dk, dv, dvp)
    LA.scan(ctx, qf, kf, vf, decay, "token", walked, scanned, heads, dk, dvp, dk ** -0.5)
    far = {"chunked": 0.0, "scan": 0.0}
    at = 0
    for i, n in enumerate(lens):
        for h in range(heads):
            part = lambda col, d: u[at: at + n, col + h * d: col + (h + 1) * d].double().cpu()
            q, k, v = part(0, dk) * dk ** -0.5, part(kd, dk), part(2 * kd, dv)
            a64, b64 = la[at: at + n, h].double().exp().cpu(), b[at: at + n, h].double().cpu()
            S0 = start[i + 1, h].double().cpu()
            want, S, norm = _recurrence(q, k, v, a64, b64, S0[:, :dv], S0[:, dv])
            size, _, _ = _recurrence(q.abs(), k.abs(), v.abs(), a64, b64, S0[:, :dv].abs(), S0[:, dv].abs())
            for name, got, left in (("chunked", out, state), ("scan", scanned, walked)):
                mine = got.view(rows, heads, dvp)[at: at + n, h].double().cpu()
                far[name] = max(far[name], ((mine[:, : dv + 1] - want).abs() / size).max().item())
                end = left[i + 1, h].double().cpu()
                assert (end[:, :dv] - S).abs().max() <= 1e-5 * S.abs().max() and (end[:, dv] - norm).abs().max() <= 1e-5 * norm.abs().max()
                assert not end[:, dv + 1:].any() and not mine[:, dv + 1:].any()
        at += n
    assert torch.equal(state[0], start[0]) and torch.equal(state[-1], start[-1])        # slots that no request of the step holds
    # relative to the sum of the sizes of a result's terms: q . k is exact products, 16 at a time in the tensor core (which cuts
    # off each of them, 2^-23 at most), those sums added pairwise in fours and then in order in float32 (2^-24 an addition); the
    # rest is 64-bit numbers and one rounding of the result
    bound = (16 + (2 + dk / 64) / 2 + 0.5) * 2.0 ** -23
    assert far["chunked"] <= bound, (far, bound)
    print(f"mlstm heads {heads} dk {dk} dv {dv}: chunked {far['chunked']:.2e} scan {far['scan']:.2e} bound {bound:.2e}")


class _Walks:
    """One request's portion through the walk in chunks and through the scan, from a zero memory."""

    def __init__(self, heads, d, n, forget, seed):
        from bare_cuda_4gib_b200.engine.step import Workspace
        from bare_cuda_4gib_b200.kernels import lib as K, mlstm as MK
        torch.manual_seed(seed)
        self.heads, self.d, self.n = heads, d, n
        ints = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
        self.ctx = types.SimpleNamespace(seq_slot=ints([0]), seq_q_start=ints([0]), seq_q_len=ints([n]), n_seqs=1, n_tokens=n, max_q_len=n,
                                         stream=K.stream_handle(), dtype=torch.bfloat16, ws=Workspace(DEV, 2048))
        self.u = (0.9 * torch.randn(n, 4 * heads * d, device=DEV)).to(torch.bfloat16)
        self.coef = torch.empty(n, heads * 4, device=DEV)
        self.la, self.b = torch.empty(n, heads, device=DEV), torch.empty(n, heads, device=DEV)
        MK.gates(self.ctx, 0.9 * torch.randn(n, 2 * heads, device=DEV), 0, heads, torch.randn(heads, device=DEV), forget + torch.randn(heads, device=DEV),
                 15.0, torch.zeros(1, heads, device=DEV), self.coef, heads, self.la, self.b)

    def run(self, chunked):
        """(results [n, heads, d + 1], memory [heads, d, d + 1])"""
        from bare_cuda_4gib_b200.kernels import linear_attention as LA, mlstm as MK
        heads, d, n, wide = self.heads, self.d, self.n, self.heads * self.d
        state, out = torch.zeros(1, heads, d, d + 4, device=DEV), torch.empty(n, heads * (d + 4), device=DEV)
        if chunked:
            MK.chunked(self.ctx, self.u, 0, wide, 2 * wide, self.la, self.b, state, out, heads, d, d, d ** -0.5)
        else:
            qf, kf, vf = torch.empty(n, wide, device=DEV), torch.empty(n, wide, device=DEV), torch.empty(n, heads * (d + 4), device=DEV)
            decay = torch.empty(n, heads, device=DEV)
            MK.operands(self.ctx, self.u, 0, wide, 2 * wide, self.coef, qf, kf, decay, vf, heads, d, d, d + 4)
            LA.scan(self.ctx, qf, kf, vf, decay, "token", state, out, heads, d, d + 4, d ** -0.5)
        return out.view(n, heads, d + 4)[..., : d + 1], state[0, ..., : d + 1]

    def exact(self, size=False):
        """The recurrence in 64 bits; with `size` the sum of its terms' sizes."""
        f = (lambda x: x.abs()) if size else (lambda x: x)
        q, k, v = (f(self.u[:, i * self.heads * self.d: (i + 1) * self.heads * self.d].double().view(self.n, self.heads, self.d)) for i in range(3))
        v = torch.cat([v, torch.ones_like(v[..., :1])], -1)
        a, b = self.la.double().exp(), self.b.double()
        S, out = torch.zeros(self.heads, self.d, self.d + 1, dtype=torch.float64, device=DEV), []
        for t in range(self.n):
            S = a[t, :, None, None] * S + b[t, :, None, None] * k[t, :, :, None] * v[t, :, None]
            out.append(torch.einsum("hkv,hk->hv", S, q[t] * self.d ** -0.5))
        return torch.stack(out), S


@pytest.mark.parametrize("d,n,forget", [(128, 40, 0.0), (128, 300, 0.0), (128, 700, 3.0), (16, 200, 0.0)])
def test_mlstm_chunked_is_no_further_from_64_bits_than_the_scan(d, n, forget):
    """By the norm of the results, by their worst element and by the norm of the memory left behind (three inputs each)."""
    far = []
    for seed in range(3):
        walks = _Walks(16, d, n, forget, seed)
        (want, memory), (size, _) = walks.exact(), walks.exact(True)
        far.append([[((y - want).norm() / want.norm()).item(), ((y - want).abs() / size).max().item(), ((s - memory).norm() / memory.norm()).item()]
                    for y, s in (walks.run(True), walks.run(False))])
    chunked, scan = torch.tensor(far).mean(0)
    assert (chunked <= scan).all(), (chunked, scan)


def test_mlstm_chunked_keeps_infinity_and_nan_from_earlier_tokens():
    walks = _Walks(2, 128, 200, 0.0, 5)
    clean, _ = walks.run(True)
    for col, token, value in ((0, 37, float("nan")), (256, 70, float("inf")), (512, 105, float("nan")), (512 + 130, 150, float("inf"))):      # q, k, v, v
        walks.u[token, col] = value
    got, scanned = walks.run(True)[0], walks.run(False)[0]
    assert torch.equal(got[:37], clean[:37]) and torch.equal(got[38:70, 0], clean[38:70, 0])
    assert torch.equal(got[:150, 1, 1:], clean[:150, 1, 1:]) and torch.equal(got[:150, 1, 0], clean[:150, 1, 0])
    assert not torch.isfinite(got[37, 0]).any() and not torch.isfinite(got[105:, 0, 0]).any() and not torch.isfinite(got[150:, 1, 2]).any()
    assert (torch.isfinite(got) >= torch.isfinite(scanned)).all()
