"""The fixed-count CG solve of grids that fit on the chip (pcg_resident.cu) against the float64 oracle's CG
(backend-cuda.cu:1788-1824), at the edges of its split: 32 x 8-cell columns, a block's range of planes crossing from one
column into the next, one-cell and one-row remainder columns, both register variants and the ends of their ranges, periodic
axes (halo words from the far side, a column that is its own neighbour) and solids.

Tolerance: FP32 vectors, FP64 dot products and 10 iterations. An iteration rounds its four updates once each (eps = 6e-8) and
the operator about seven times; carried through 10 iterations of growing search directions (at most a factor of ten) that is
10 * 11 * 6e-8 * 10 < 1e-4 of the largest pressure.
"""
import ctypes as C
import time

import numpy as np
import pytest
import torch

import oracle as O
import scenes
import smoke_abi as abi
import smoke_b200

pytestmark = pytest.mark.gpu

SHAPES = [
    (8, 8, 8),       # one block, one plane row of a column
    (33, 9, 16),     # remainder columns of one cell and one row
    (32, 8, 40),     # a single column cut into blocks
    (40, 24, 9),     # planes of two columns in one block
    (31, 57, 23),
    (65, 41, 48),
    (96, 128, 96),   # 32 planes a block: the end of the middle variant
    (128, 128, 128), # the large variant
]


# 2 to 16 blocks run as one cluster, whatever the count; 17 do not
CLUSTERS = [(32, 8, 8 * blocks) for blocks in (2, 3, 5, 6, 7, 8, 9, 11, 13, 14, 15, 16, 17)]


@pytest.mark.parametrize("boundary", ["closed", "plume", "zout"])
@pytest.mark.parametrize("shape", SHAPES, ids=["x".join(map(str, s)) for s in SHAPES])
@pytest.mark.parametrize("reduction", [abi.REDUCTION_FP32, abi.REDUCTION_FP64], ids=["fp32", "fp64"])
def test_fixed_cg_on_chip_matches_oracle(smoke_lib, cuda_stream, shape, boundary, reduction):
    check_against_oracle(smoke_lib, cuda_stream, shape, boundary, reduction)


@pytest.mark.parametrize("shape", CLUSTERS, ids=["x".join(map(str, s)) for s in CLUSTERS])
def test_fixed_cg_in_one_cluster_matches_oracle(smoke_lib, cuda_stream, shape):
    check_against_oracle(smoke_lib, cuda_stream, shape, "plume", abi.REDUCTION_FP32)


# 69, 70 (the most that a block holds) and 71 planes a block on 148 SMs; the last is the streaming kernel's
@pytest.mark.parametrize("reduction", [abi.REDUCTION_FP32, abi.REDUCTION_FP64], ids=["fp32", "fp64"])
@pytest.mark.parametrize("nz,on_chip", [(127, True), (128, True), (130, False)])
def test_the_largest_grids_on_the_chip(smoke_lib, cuda_stream, nz, on_chip, reduction):
    check_against_oracle(smoke_lib, cuda_stream, (128, 160, nz), "plume", reduction)
    cfg = scenes.make_config(128, 160, nz, boundary="plume", pressure_iterations=10)
    sim = smoke_b200.Simulation(smoke_lib, cfg, cuda_stream)
    sim.set_solver(abi.SOLVER_FIXED_CG, reduction)
    st = abi.SolverStatus()
    # the hook takes the solves that run on the chip; a block that does not exist withholds nothing
    rc = smoke_lib.lib.smoke_b200_test_exchange_timeout_cuda(sim.handle, 1 << 20, 1, 1000, C.byref(st))
    sim.close()
    assert (rc == abi.RESULT_OK) == on_chip
    assert not on_chip or st.status == abi.SOLVE_ITERATION_CAP


def check_against_oracle(smoke_lib, cuda_stream, shape, boundary, reduction):
    cfg = scenes.make_config(*shape, boundary=boundary, mode=abi.LINEAR, pressure_iterations=10)
    inp = scenes.random_inputs(cfg, seed=sum(shape), solids=shape[0] != 32)
    sim = smoke_b200.Simulation(smoke_lib, cfg, cuda_stream)
    keep = scenes.load_gpu(sim, inp)
    sim.set_solver(abi.SOLVER_FIXED_CG, reduction)
    with torch.cuda.stream(cuda_stream):
        sim.step_stages(abi.STAGE_PRESSURE)
    rhs = sim.snapshot([abi.VIEW_FLOW_PRESSURE_RHS])["pressure_rhs"]
    p = sim.snapshot([abi.VIEW_FLOW_PRESSURE])["pressure"]
    with torch.cuda.stream(cuda_stream):
        sim.solve_pressure()  # the next launch's words carry other tags in the same buffers
    again = sim.snapshot([abi.VIEW_FLOW_PRESSURE])["pressure"]
    status = sim.solver_status()
    sim.close()
    del keep
    x, _ = O.solve_pressure(cfg, inp["occupancy"], rhs, bits=64, mode=0)
    assert status.iterations == 10 and status.status == abi.SOLVE_ITERATION_CAP
    assert np.array_equal(p, again)
    assert scenes.rel_err(p, x) < 1e-4


# the iterations whose halo waits run out: the first, one in the middle and the last, whose sums alone tell the others
@pytest.mark.parametrize("exchange", [1, 5, 10])
@pytest.mark.parametrize("shape,block", [((32, 8, 40), 2), ((48, 40, 32), 1), ((96, 96, 96), 70)], ids=["cluster", "grid", "planes24"])
def test_halo_wait_that_runs_out_aborts_the_solve(smoke_lib, cuda_stream, shape, block, exchange):
    """A block that never gets its neighbours' faces of one exchange: its bounded waits run out, every block leaves, the
    status says so, and the next solve on the context gives the bits of the one before."""
    cfg = scenes.make_config(*shape, boundary="plume", mode=abi.LINEAR, pressure_iterations=10)
    inp = scenes.random_inputs(cfg, seed=sum(shape), solids=False)
    sim = smoke_b200.Simulation(smoke_lib, cfg, cuda_stream)
    keep = scenes.load_gpu(sim, inp)
    sim.set_solver(abi.SOLVER_FIXED_CG, abi.REDUCTION_FP32)
    with torch.cuda.stream(cuda_stream):
        sim.step_stages(abi.STAGE_PRESSURE)
    p = sim.snapshot([abi.VIEW_FLOW_PRESSURE])["pressure"]
    st = abi.SolverStatus()
    hook = smoke_lib.lib.smoke_b200_test_exchange_timeout_cuda
    t0 = time.perf_counter()
    assert hook(sim.handle, block, exchange, 100, C.byref(st)) == abi.RESULT_OK
    waited = time.perf_counter() - t0
    assert st.status == abi.SOLVE_BARRIER_TIMEOUT, st.status
    assert 0.05 < waited < 5.0, waited
    with torch.cuda.stream(cuda_stream):
        sim.solve_pressure()
    again = sim.snapshot([abi.VIEW_FLOW_PRESSURE])["pressure"]
    status = sim.solver_status()
    assert status.iterations == 10 and status.status == abi.SOLVE_ITERATION_CAP
    assert np.array_equal(p, again)
    assert hook(sim.handle, block, 0, 100, C.byref(st)) == abi.RESULT_BACKEND_FAILURE
    sim.set_solver(abi.SOLVER_JACOBI_PCG, abi.REDUCTION_FP64, max_iterations=100, tolerance=1e-5)
    assert hook(sim.handle, block, 1, 100, C.byref(st)) == abi.RESULT_BACKEND_FAILURE  # no exchange of faces there
    sim.close()
    del keep


@pytest.mark.parametrize("shape,boundary", [((8, 8, 8), "closed"), ((32, 8, 40), "plume"), ((40, 24, 9), "zout"), ((33, 41, 37), "closed"), ((64, 64, 64), "plume")])
@pytest.mark.parametrize("reduction", [abi.REDUCTION_FP32, abi.REDUCTION_FP64], ids=["fp32", "fp64"])
def test_the_two_kernels_agree_after_64_iterations(smoke_lib, cuda_stream, shape, boundary, reduction):
    """The allocation-free solve runs the streaming kernel on the same system. The kernels' totals differ by the order in which up
    to 148 FP64 partials are added (2^-53 each), which changes alpha or beta, rounded to FP32, only where the total lies that
    close to a rounding boundary. Were one to flip in every one of 64 iterations (2^-24 of a step), with the growth by a factor
    of ten allowed above, that would be 64 * 6e-8 * 10 < 1e-4 of the largest pressure."""
    cfg = scenes.make_config(*shape, boundary=boundary, mode=abi.LINEAR, pressure_iterations=64)
    inp = scenes.random_inputs(cfg, seed=sum(shape), solids=False)
    sim = smoke_b200.Simulation(smoke_lib, cfg, cuda_stream)
    keep = scenes.load_gpu(sim, inp)
    sim.set_solver(abi.SOLVER_FIXED_CG, reduction)
    with torch.cuda.stream(cuda_stream):
        sim.step_stages(abi.STAGE_PRESSURE)
        rhs = sim.view(abi.VIEW_FLOW_PRESSURE_RHS).clone()
    p = sim.snapshot([abi.VIEW_FLOW_PRESSURE])["pressure"]
    sim.close()
    del keep
    solve = smoke_lib.lib.smoke_b200_solve_pressure_noalloc_cuda
    solve.argtypes = [C.POINTER(abi.Config), C.c_void_p, C.c_void_p, C.c_void_p, C.POINTER(abi.SolverDesc), C.c_void_p, C.POINTER(abi.SolverStatus)]
    solve.restype = C.c_int
    out, st, desc = torch.empty_like(rhs), abi.SolverStatus(), abi.SolverDesc(abi.SOLVER_FIXED_CG, reduction, 500, 1e-5, 0, 0)
    torch.cuda.synchronize()
    rc = solve(C.byref(cfg), None, C.c_void_p(rhs.data_ptr()), C.c_void_p(out.data_ptr()), C.byref(desc), C.c_void_p(cuda_stream.cuda_stream), C.byref(st))
    assert rc == abi.RESULT_OK and st.iterations == 64
    assert scenes.rel_err(p, out.cpu().numpy()) < 1e-4
