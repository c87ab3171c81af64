"""The pressure stage just above and below the sizes at which kernels change their split: columns of cells per thread in the
face-force, right-hand-side and projection kernels (from 600 000 cells with planes of 4096), four rows per thread in the
level-0 multigrid passes (from 512 000 cells), paired children in the prolongation (even x extent), and the table of the
block levels. Extents leave remainders of every tile. A wrong face, right-hand side or gradient anywhere leaves a
divergence of the order of max|u| / h in its cell, so the check is the divergence of the projected faces, formed in float64.
Its bound: the solve is held to a true residual of 1e-9, and each of a cell's six faces carries one FP32 rounding of its
value (6 x 2^-24 = 3.6e-7 of max|u| / h) and one of the gradient subtracted from a face before it was projected, which may
be several times larger; 1e-5 leaves a factor of 28 for that."""
import numpy as np
import pytest
import torch

import scenes
import smoke_abi as abi
import smoke_b200

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,nz,boundary,solids", [(97, 81, 83, "plume", True), (98, 83, 77, "closed", False), (70, 131, 69, "mixed", True), (79, 81, 79, "zout", False), (20, 33, 950, "closed", False)])
def test_projected_faces_are_free_of_divergence(smoke_lib, cuda_stream, nx, ny, nz, boundary, solids):
    cfg = scenes.make_config(nx, ny, nz, boundary=boundary)
    inp = scenes.random_inputs(cfg, seed=31, solids=solids)
    sim = smoke_b200.Simulation(smoke_lib, cfg, cuda_stream)
    keep = scenes.load_gpu(sim, inp)
    sim.set_solver(abi.SOLVER_MG_FCG, abi.REDUCTION_FP64, max_iterations=400, tolerance=1e-9, refinement=6)
    with torch.cuda.stream(cuda_stream):
        sim.step()
    status = sim.solver_status()
    with torch.cuda.stream(cuda_stream):
        faces = [t.clone() for t in sim.face_velocity(0)]
    cuda_stream.synchronize()
    sim.close()
    del keep
    assert status.status == abi.SOLVE_CONVERGED and status.true_relative_residual <= 1e-9
    u, v, w = (t.cpu().numpy().astype(np.float64) for t in faces)
    div = u[:, :, 1:] - u[:, :, :-1] + v[:, 1:, :] - v[:, :-1, :] + w[1:, :, :] - w[:-1, :, :]
    fluid = inp["occupancy"] == 0
    # an OUTFLOW face copies its interior neighbour (backend-cuda.cu:1023-1024), so the cells behind it keep a divergence
    for axis, name in ((2, "x"), (1, "y"), (0, "z")):
        for side, index in (("minus", 0), ("plus", -1)):
            if getattr(cfg.flow_boundary, f"{name}_{side}").type == abi.OUTFLOW:
                fluid[(slice(None),) * axis + (index,)] = False
    fluid[np.unravel_index(np.argmax(inp["occupancy"] == 0), fluid.shape)] = False  # the anchor's equation is p = 0
    scale = max(np.abs(f).max() for f in (u, v, w))
    assert np.isfinite(div).all() and scale > 0
    assert np.abs(div[fluid]).max() / scale <= 1e-5, np.abs(div[fluid]).max() / scale
