"""The training tail where its tensors are not each by themselves: one tensor in two roles, one tensor under two
names (it steps once per name, in turn), each against the form that takes the tensors in turn (chosen by a
storage that is not 16-byte aligned).  And the streaming form where a block takes two and four steps through its
tensor, with a remainder of rows.  The bound is that of the tail's other tests."""
import pytest
import torch

import test_gpu_tail_forms as forms

pytestmark = pytest.mark.gpu


def _run(n, shared, dev):
    from ray_gauss_b200.train_tail import FusedTrainTail, LrSchedule
    got = []
    for offset in (0, 1):
        w = dict(positions=(3,), scales=(3,), rgb=(3,), sh=(3, 15))
        p, g = forms._tensors(n, offset, dev, w), forms._tensors(n, 0, dev, w)
        roles = dict(positions="positions", scales="scales")
        if shared == "roles":
            roles["lobe_axis"] = "scales"
        else:
            p["tied"], g["tied"] = p["sh"], g["sh"] * 0.5
        tail = FusedTrainTail(p, {k: LrSchedule(1e-2) for k in p}, roles=roles, normalize_lobe_axis=shared == "roles",
                              max_scale=0.5)
        floor = torch.linspace(-1.0, 0.2, n, device=dev)
        for _ in range(3):
            tail.step(min_scale=floor, grads=g)
        got.append({**{"p." + k: v for k, v in tail.params.items()}, **{"m." + k: v for k, v in tail.exp_avg.items()},
                    **tail.stats})
    return got


@pytest.mark.parametrize("shared", ["roles", "tensor"])
@pytest.mark.parametrize("n", [1023, 5003])
def test_shared_tensors_step_in_turn(cuda, n, shared):
    got = _run(n, shared, cuda)
    for k in got[0]:
        assert torch.allclose(got[0][k], got[1][k], rtol=2e-6, atol=2e-7), k


@pytest.mark.parametrize("n", [60_003, 130_001])     # 94 floats per Gaussian: two and four steps per block
def test_several_steps_per_block(cuda, n):
    forms.test_streaming_form_equals_the_unaligned_form(cuda, n, forms.WIDTHS)
