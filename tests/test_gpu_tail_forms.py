"""The streaming form of the training tail against its form for unaligned tensors (held to torch's Adam by
the tail's own tests), at the sizes where its rows and remainders can go wrong.  The bound is that of
those tests."""
import pytest
import torch

pytestmark = pytest.mark.gpu
WIDTHS = dict(positions=(3,), densities=(), scales=(3,), quaternions=(4,), rgb=(3,), sh=(3, 15), sg=(3, 5),
              bandwidth=(5,), axis=(5, 3))


NARROW = {k: WIDTHS[k] for k in ("positions", "densities", "scales", "quaternions", "rgb", "axis")}


def _tensors(n, offset, dev, widths):
    """Random tensors whose storage starts `offset` floats after a 16-byte boundary."""
    gen = torch.Generator(device="cpu").manual_seed(n)
    out = {}
    for k, sh in widths.items():
        flat = torch.empty(offset + n * int(torch.Size(sh).numel()), device=dev)
        t = flat[offset:].view((n,) + sh)
        t.copy_(torch.randn((n,) + sh, generator=gen))
        out[k] = t
    return out


@pytest.mark.parametrize("n,widths", [(n, WIDTHS) for n in (1, 3, 4, 5, 1023, 4096, 5003)] +
                         [(n, NARROW) for n in (49_999, 50_000, 50_001)])   # narrow rows: whole blocks from 50k on
def test_streaming_form_equals_the_unaligned_form(cuda, n, widths):
    from ray_gauss_b200.train_tail import FusedTrainTail, LrSchedule
    got = []
    for offset in (0, 1):
        p, g = _tensors(n, offset, cuda, widths), _tensors(n, 0, cuda, widths)
        g["positions"][::2] = 0.0
        if offset == 0:
            p["quaternions"][0] = 0.0
        else:                                       # quaternions must be aligned in either form
            p["quaternions"] = p["quaternions"].clone()
            p["quaternions"][0] = 0.0
        p["axis"][n // 2] = 0.0
        roles = dict(positions="positions", densities="densities", scales="scales", quaternions="quaternions",
                     lobe_axis="axis")
        tail = FusedTrainTail(p, {k: LrSchedule(1e-2) for k in p}, roles=roles, normalize_lobe_axis=True, max_scale=0.5)
        floor = torch.linspace(-1.0, 0.2, n, device=cuda)
        for it in range(3):
            if it == 2:
                g["rgb"] = g["axis"] = None          # no step; the axes are normalised all the same
            tail.step(min_scale=floor, grads=g)
        got.append({**{"p." + k: v for k, v in tail.params.items()}, **{"m." + k: v for k, v in tail.exp_avg.items()},
                    **{"v." + k: v for k, v in tail.exp_avg_sq.items()}, **tail.stats})
    for k in got[0]:
        assert torch.allclose(got[0][k], got[1][k], rtol=2e-6, atol=2e-7), k
