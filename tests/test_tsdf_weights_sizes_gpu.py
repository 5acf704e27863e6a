"""Warp weights of voxels on both sides of the volume where a thread takes one voxel or four: against numpy's arithmetic in
binary32 within the library's exponential, equal for equal voxels bit for bit, and nothing written where there are no
neighbours."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [4, 8])
def test_weights_do_not_depend_on_the_size(k):
    from volumefusion_gb300 import af
    g = torch.Generator(device="cuda").manual_seed(k)
    n, m, big = 50, 70001, 3000000
    cnt = torch.randint(0, k + 1, (m,), generator=g, device="cuda", dtype=torch.int32)
    cnt[torch.rand(m, generator=g, device="cuda") < 0.6] = 0
    idx = torch.randint(0, n, (m, k), generator=g, device="cuda", dtype=torch.int32)
    dist = 0.04 * torch.rand((m, k), generator=g, device="cuda")
    radii = 0.01 + 0.02 * torch.rand(n, generator=g, device="cuda")
    out = []
    for S in (m, big - 1, big, big + 77):
        w = torch.full((S, k), 7.0, device="cuda")
        c = torch.zeros(S, dtype=torch.int32, device="cuda")
        i, d = torch.zeros((S, k), dtype=torch.int32, device="cuda"), torch.zeros((S, k), device="cuda")
        c[-m:], i[-m:], d[-m:] = cnt, idx, dist
        af.runComputeTsdfWarpWeightsKernel(w, radii, i, d, c, S)
        assert bool((w[:S - m] == 7).all())
        out.append(w[-m:].clone())
    assert all(torch.equal(o, out[0]) for o in out)
    w = out[0].cpu().numpy()
    c, d, r = cnt.cpu().numpy(), dist.cpu().numpy().astype(np.float64), radii.cpu().numpy().astype(np.float64)[idx.cpu().numpy()]
    e = np.where(np.arange(k)[None] < c[:, None], np.exp(-d * d / (2 * r * r)), 0.0)
    s = e.sum(1, keepdims=True)
    want = np.where(c[:, None] > 0, e / np.where(s > 0, s, 1), 7.0)
    # k + 3 roundings and one exponential of at most 4 ulp on either side of the quotient
    assert np.abs(w - want).max() <= 2 * (k + 8) * 2.0 ** -24 * 7
