"""cross_correlate_particle_stack (core_refine_template.py:771-895): the oracle
against vectors recorded from the reference's own function (CPU), the device
path against both (GPU).  Tolerance: 1e-4 of the largest |correlation| (FP32
FFTs of different factorisations)."""

import os

import numpy as np
import pytest
import torch

from oracle import ref_refine_template as orr

GOLD = np.load(os.path.join(os.path.dirname(__file__), "golden", "xcorr_small.npz"))


def _case(name):
    return (torch.from_numpy(GOLD[f"{name}/stack"]), torch.from_numpy(GOLD[f"{name}/template_dft"]),
            torch.from_numpy(GOLD[f"{name}/rot"]), torch.from_numpy(GOLD[f"{name}/filters"]))


def _close(got, ref, tol=1e-4):
    ref = np.asarray(ref)
    err = np.abs(np.asarray(got) - ref).max() / np.abs(ref).max()
    assert err <= tol, f"relative error {err:.3e}"


@pytest.mark.parametrize("name", ["x1", "x2"])
@pytest.mark.parametrize("mode", ["valid", "same"])
def test_oracle_matches_reference(name, mode):
    got = orr.cross_correlate_particle_stack_cpu(*_case(name), mode=mode)
    _close(got.numpy(), GOLD[f"{name}/{mode}"], 1e-5)


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["x1", "x2"])
@pytest.mark.parametrize("mode", ["valid", "same"])
@pytest.mark.parametrize("batch", [1, 2, -1])
def test_device_matches_reference(name, mode, batch):
    from leopard_em_gb300.backend import cross_correlate_particle_stack

    got = cross_correlate_particle_stack(*_case(name), mode=mode, batch_size=batch)
    assert got.device.type == "cpu" and tuple(got.shape) == GOLD[f"{name}/{mode}"].shape
    _close(got.numpy(), GOLD[f"{name}/{mode}"])


@pytest.mark.gpu
def test_device_matches_oracle_refine_size():
    """288^2 crops with a 256^3 template (the refinement configuration's shapes)."""
    from leopard_em_gb300 import synthetic as sy
    from leopard_em_gb300.backend import cross_correlate_particle_stack

    cfg = sy.RefineConfig(crop=288, template_size=256, n_blobs=300, blob_radius=80.0)
    kw, _ = sy.make_refine_workload(cfg, 3)
    rot = sy.axis_angle_rotations(torch.tensor([[0.0, 0.0, 1.0]] * 3), torch.tensor([0.1, 0.7, 2.0]))
    pf = kw["projective_filters"]
    ps = kw["particle_stack_dft"].clone()
    ps[:, 0, 0] = 5.0 + 0j  # non-zero DC: the term the search path zeroes
    got = cross_correlate_particle_stack(ps.cuda(), kw["template_dft"], rot.float(), pf, mode="valid")
    assert got.is_cuda
    ref = orr.cross_correlate_particle_stack_cpu(ps, kw["template_dft"], rot.float(), pf, mode="valid")
    _close(got.cpu().numpy(), ref.numpy())


@pytest.mark.gpu
def test_device_argument_errors():
    from leopard_em_gb300.backend import cross_correlate_particle_stack

    ps, t, r, f = _case("x1")
    with pytest.raises(ValueError):
        cross_correlate_particle_stack(ps, t, r, f, mode="full")
    with pytest.raises(ValueError):
        cross_correlate_particle_stack(ps, t, r[:2], f)
    with pytest.raises(ValueError):
        cross_correlate_particle_stack(ps, t, r, f, mag_matrix=torch.eye(2))


@pytest.mark.gpu
@pytest.mark.parametrize("H,W,d,mode", [(64, 64, 48, "valid"), (128, 128, 96, "same"), (256, 256, 192, "valid"),
                                        (288, 288, 256, "same"), (288, 288, 64, "same")])
def test_device_reads_the_particles_own_rows(H, W, d, mode):
    """Images of W/2 + 1 columns read in place by the short column passes; projections normalised there or before."""
    test_device_matches_oracle_register_column_lengths(H, W, d, mode)


@pytest.mark.gpu
@pytest.mark.parametrize("H,W,d,mode", [(576, 80, 48, "same"), (1024, 64, 32, "valid"), (2048, 48, 48, "same")])
def test_device_matches_oracle_register_column_lengths(H, W, d, mode):
    """The register column passes with another image for each correlogram."""
    from leopard_em_gb300.backend import cross_correlate_particle_stack

    g = torch.Generator().manual_seed(H + d)
    ps = torch.fft.rfft2(torch.randn((3, H, W), generator=g))
    vol = torch.fft.fftshift(torch.fft.rfftn(torch.randn((d, d, d), generator=g)), dim=(0, 1))
    rot = torch.linalg.qr(torch.randn((3, 3, 3), generator=g, dtype=torch.float64))[0].float()
    rot *= torch.linalg.det(rot)[:, None, None].sign()
    pf = torch.rand((3, d, d // 2 + 1), generator=g) + 0.5
    got = cross_correlate_particle_stack(ps, vol, rot, pf, mode=mode)
    ref = orr.cross_correlate_particle_stack_cpu(ps, vol, rot, pf, mode=mode)
    _close(got.numpy(), ref.numpy())


@pytest.mark.gpu
@pytest.mark.parametrize("H,d", [(64, 48), (128, 96), (256, 192), (288, 256), (512, 96)])
def test_particles_at_an_odd_storage_offset(H, d):
    """The column passes read the caller's rows: a stack that starts 8 bytes off a 16-byte line gives the same bits."""
    from leopard_em_gb300.backend import cross_correlate_particle_stack

    g = torch.Generator().manual_seed(H)
    ps = torch.fft.rfft2(torch.randn((3, H, H), generator=g)).cuda()
    vol = torch.fft.fftshift(torch.fft.rfftn(torch.randn((d, d, d), generator=g)), dim=(0, 1)).cuda()
    rot = torch.linalg.qr(torch.randn((3, 3, 3), generator=g, dtype=torch.float64))[0].float().cuda()
    pf = (torch.rand((3, d, d // 2 + 1), generator=g) + 0.5).cuda()
    buf = torch.empty(ps.numel() + 1, dtype=ps.dtype, device=ps.device)
    odd = buf[1:].view(ps.shape).copy_(ps)
    assert odd.data_ptr() % 16 == 8 and odd.is_contiguous()
    assert torch.equal(cross_correlate_particle_stack(odd, vol, rot, pf), cross_correlate_particle_stack(ps, vol, rot, pf))
