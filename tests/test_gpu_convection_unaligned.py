"""Convection of device fields at 8-byte offsets runs the line kernel at every
order, even ones with single loads in place of pairs: bitwise what the same
fields give on 16-byte boundaries, for the whole mesh and a part of it."""
import numpy as np
import pytest

from ssenss_b200.mesh import box_mesh, channel_mesh

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", range(2, 13))
@pytest.mark.parametrize("mesh", ["box", "channel"])
def test_offset_fields_are_bitwise(mesh, n, gpu_ctx_factory):
    import torch
    m = box_mesh((3, 3, 3)) if mesh == "box" else channel_mesh((4, 3, 3), seed=7)
    ctx = gpu_ctx_factory(m, n)
    rng = np.random.default_rng(n)
    u, v = (torch.from_numpy(rng.standard_normal((3, m.nel, n, n, n))).cuda() for _ in range(2))

    def offset(x):
        raw = torch.zeros(x.numel() + 1, dtype=torch.float64, device="cuda")
        y = raw[1:].view(x.shape)
        y.copy_(x)
        return y

    for a, b in ((u, v), (u, u)):
        ao = offset(a)
        bo = ao if b is a else offset(b)
        out, out_o = torch.empty_like(u), offset(torch.zeros_like(u))
        torch.cuda.synchronize()
        ctx.convection_operator(a, b, out)
        ctx.convection_operator(ao, bo, out_o)
        assert torch.equal(out, out_o)
        part = [x[:, 2:7].contiguous() for x in (a, b)]
        po = offset(part[0])
        qo = po if b is a else offset(part[1])
        torch.cuda.synchronize()
        got = ctx.convection_elements(2, po, qo, torch.empty_like(part[0]))
        assert torch.equal(got, out[:, 2:7])
    ctx.close()
