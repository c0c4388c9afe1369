"""The x pass's scaling by maps against the uniform material, bit for bit."""
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _m(N, seed):
    return torch.randn((3,) + N[::-1], device="cuda", generator=torch.Generator("cuda").manual_seed(seed))


@pytest.mark.parametrize("N,pbc", [((39, 9, 1), (0, 0, 0)), ((64, 20, 3), (0, 0, 0)), ((250, 13, 1), (0, 0, 0)),
                                   ((600, 6, 2), (0, 0, 0)), ((96, 10, 1), (1, 0, 0)), ((512, 5, 1), (2, 0, 0))])
def test_maps_equal_uniform_material(N, pbc):
    """Scaling by powers of two is exact, so MU0*Ms*vol*m has the same bits whichever map carries the factors."""
    from umagnus_b200 import opencl
    plan = opencl.NewNewellDemag(N, pbc, (2e-9, 2e-9, 2e-9))
    g = torch.Generator("cuda").manual_seed(5)
    w = 2.0 ** torch.randint(-2, 2, N[::-1], device="cuda", generator=g).float()
    w[torch.rand(N[::-1], device="cuda", generator=g) < 0.2] = 0.0
    ms = 8e5 * 2.0 ** torch.randint(-1, 2, N[::-1], device="cuda", generator=g).float()
    m = _m(N, 1)
    got, want = torch.empty_like(m), torch.empty_like(m)
    for vol, Ms, scale in ((w, 8e5, w), (None, opencl.MSlice(ms), ms / 8e5), (w, opencl.MSlice(ms), w * (ms / 8e5))):
        plan.Exec(got, m, vol, Ms)
        plan.Exec(want, (m * scale).contiguous(), None, 8e5)
        assert torch.equal(got, want)
