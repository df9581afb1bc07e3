"""Host decoding of the refinement's results against the FP64 torch composition."""

import numpy as np
import pytest
import torch

from leopard_em_gb300 import rotations as rot


def _words(n, seed, given):
    g = torch.Generator().manual_seed(seed)
    words = torch.zeros((n, 13), dtype=torch.int32)
    f = words.view(torch.float32)
    f[:, 0], f[:, 1] = torch.randn(n, generator=g), torch.randn(n, generator=g)
    words[:, 2:5] = torch.randint(0, 33, (n, 3), generator=g, dtype=torch.int32)
    f[:, 5:7] = torch.randn((n, 2), generator=g)
    f[:, 7:10] = 3 * torch.randn((n, 3), generator=g)
    # theta stays off the poles, where the first and the last angle are one
    pose = torch.rand((n, 3), generator=g, dtype=torch.float64) * torch.tensor([360.0, 140.0, 360.0]) + torch.tensor(
        [0.0, 20.0, 0.0])
    f[:, 10:13] = pose.float()
    if n > 1:
        f[1, 7:10] = 0.0  # no offset
    return words, pose if given else None


@pytest.mark.parametrize("n,given", [(0, False), (1, False), (2, True), (65, False), (65, True)])
def test_decode_matches_torch(n, given):
    from leopard_em_gb300.backend.core_refine_template import decode_refine_results

    words, pose = _words(n, n, given)
    f = words.view(torch.float32)
    got = decode_refine_results(words, pose, 33, 30)
    e = rot.combine_euler_angles(f[:, 7:10].double(), f[:, 10:13].double() if pose is None else pose).float()
    e = torch.where(e < 0, e + torch.tensor([360.0, 180.0, 360.0]), e)
    # FP64 compositions of one formula, rounded to FP32: one unit in the last place of 360
    assert np.allclose(got["refined_euler_angles"].numpy(), e.numpy(), rtol=0, atol=4e-5)
    assert torch.equal(got["refined_pos_y"], words[:, 2].long() - 16)
    assert torch.equal(got["refined_pos_x"], words[:, 3].long() - 15)
    assert torch.equal(got["angle_idx"], words[:, 4].long())
    for k, w in (("refined_z_score", 0), ("refined_cross_correlation", 1), ("refined_defocus_offset", 5),
                 ("refined_pixel_size_offset", 6)):
        assert torch.equal(got[k], f[:, w])


@pytest.mark.parametrize("theta", [0.0, 180.0])
def test_decode_at_the_poles(theta):
    """No offset on a pole: the composition's zeros keep torch's signs."""
    from leopard_em_gb300.backend.core_refine_template import decode_refine_results

    words = torch.zeros((1, 13), dtype=torch.int32)
    words.view(torch.float32)[0, 11] = theta
    f = words.view(torch.float32)
    e = rot.combine_euler_angles(f[:, 7:10].double(), f[:, 10:13].double()).float()
    e = torch.where(e < 0, e + torch.tensor([360.0, 180.0, 360.0]), e)
    assert torch.equal(decode_refine_results(words, None, 33, 33)["refined_euler_angles"], e)


@pytest.mark.parametrize("change", [{"euler_angles": (3, 3)}, {"euler_angles": (1, 3)}, {"euler_angles": (2, 2)},
                                    {"euler_angle_offsets": (5, 1)}, {"euler_angle_offsets": (5,)},
                                    {"defocus_u": (1,)}, {"defocus_angle": (0,)}])
def test_poses_and_offsets_of_another_shape_are_refused(change):
    """Before any device work: the decoding no longer runs through torch operations that refuse them."""
    from leopard_em_gb300.backend import core_refine_template

    shapes = {"euler_angles": (2, 3), "euler_angle_offsets": (5, 3), "defocus_offsets": (1,), "defocus_u": (2,),
              "defocus_v": (2,), "defocus_angle": (2,), "pixel_size_offsets": (1,), "corr_mean": (2, 17, 17),
              "corr_std": (2, 17, 17), "projective_filters": (2, 48, 25)}
    kw = {k: torch.zeros(change.get(k, s)) for k, s in shapes.items()}
    kw["particle_stack_dft"] = torch.zeros((2, 64, 33), dtype=torch.complex64)
    kw["template_dft"] = torch.zeros((48, 48, 25), dtype=torch.complex64)
    ctf = {"voltage": 300.0, "spherical_aberration": 2.7, "amplitude_contrast_ratio": 0.07, "ctf_B_factor": 0.0,
           "phase_shift": 0.0, "pixel_size": 1.0}
    with pytest.raises(ValueError, match=next(iter(change))):
        core_refine_template(**kw, ctf_kwargs=ctf, device=torch.device("cuda:0"))
