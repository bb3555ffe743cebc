"""Muon's element-wise kernels (one launch on each side of the orthogonalisation) against the separate PyTorch operations,
which they round like: aligned and unaligned matrices, clipping, skipped steps."""
import math

import pytest
import torch

from ttcd_b200 import ops
from ttcd_b200.train.muon import MuonParam, _fused_ok, muon_update_many

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("shapes", [[(128, 128)], [(136, 168), (136, 168)], [(128, 256), (256, 128), (128, 256)], [(1024, 136)]])
@pytest.mark.parametrize("coef,skip,nesterov", [(None, None, True), (0.37, 0, True), (0.37, 1, True), (None, 0, False)])
def test_fused_muon_update(shapes, coef, skip, nesterov):
    torch.manual_seed(len(shapes))
    lr, wd, mom = 0.02, 0.1, 0.95
    coef_t = None if coef is None else torch.tensor([coef], device=DEV)
    skip_t = None if skip is None else torch.tensor([skip], dtype=torch.int32, device=DEV)
    params = []
    for i, s in enumerate(shapes):
        n = math.prod(s)
        mp = MuonParam(str(i), torch.nn.Parameter(torch.zeros(s, device=DEV)), 0, 0)
        off = i % 2                                          # every other matrix starts 4 bytes off: the scalar kernels
        mp.master, mp.momentum, mp.grad32 = (torch.randn(n + off, device=DEV)[off:] for _ in range(3))
        assert _fused_ok(mp, coef_t, skip_t, None)
        params.append(mp)
    before = [(mp.master.clone(), mp.momentum.clone()) for mp in params]
    places = {id(mp): torch.empty(mp.param.numel(), dtype=torch.bfloat16, device=DEV) for mp in params}
    published = muon_update_many(params, lr, wd, mom, coef_t, nesterov, skip_t, publish=lambda mp: places[id(mp)])
    assert published == {id(mp) for mp in params}
    for s in set(shapes):                                    # matrices of one shape are orthogonalised together
        group = [i for i, t in enumerate(shapes) if t == s]
        news, gs = [], []
        for i in group:
            g = params[i].grad32 if coef is None else params[i].grad32 * coef_t
            new = before[i][1] * mom + g
            news.append(new)
            gs.append((g.add(new, alpha=mom) if nesterov else new).view(s))
        u = ops.newton_schulz(torch.stack(gs)).float()
        for j, i in enumerate(group):
            want = (before[i][0] * (1.0 - lr * wd)).add_(u[j].reshape(-1), alpha=-lr * 0.2 * math.sqrt(max(s)))
            if skip:
                assert torch.equal(params[i].master, before[i][0]) and torch.equal(params[i].momentum, before[i][1])
            else:
                assert torch.equal(params[i].momentum, news[j])
                assert (params[i].master - want).abs().max() <= 2.0 ** -22 * want.abs().max()     # one fp32 rounding apart
            assert torch.equal(places[id(params[i])], params[i].master.bfloat16())
