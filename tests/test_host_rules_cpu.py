"""The host side of lbm_iterate without a GPU: what it launches, and what it does when the runtime
refuses."""

from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from tests.fake_runtime import STORAGE, FakeSim, load


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    return load(tmp_path_factory.mktemp("fake"))


@pytest.mark.parametrize("counts,storage,kernel", [((64, 64), "f32", "aa_resident_kernel"),
                                                   ((200, 150), "f16", "aa_resident_kernel"),
                                                   ((64, 64, 256), "f16", "aa_tma_kernel")])
def test_kernels_are_set_up_on_every_device(lib, counts, storage, kernel):
    """Shared memory above 48 KB is opted into per device: a simulation on a second GPU of the
    process runs as one on the first, in either order and again."""
    for device in (1, 0, 1):
        sim = FakeSim(lib, counts, storage=storage, device=device)
        sim.check(sim.iterate(20))
        launched = sim.launched()
        assert launched and all(d == device and kernel in name for d, name in launched)
        sim.close()


def test_ensemble_and_closure_are_set_up_on_every_device(lib):
    nx, ny = 40, 70
    params = np.zeros(10752, np.float32)
    fields = [np.zeros(nx * ny * 2, np.float32) for _ in range(4)]
    p = lambda a: C.c_void_p(a.ctypes.data)  # noqa: E731
    for device in (1, 0):
        lib.fake_set_device(device)
        h = C.c_void_p()
        counts = (C.c_int64 * 2)(40000, 128)  # too large for the flat kernel: rows, staged
        om = (C.c_float * 1)(1.6)
        assert lib.lbm_ensemble_create(1, counts, 0, om, om, 0, C.byref(h)) == 0
        assert lib.lbm_ensemble_iterate(h, C.c_int64(2), 0) == 0, lib.lbm_last_error()
        lib.lbm_ensemble_destroy(h)
        lib.fake_take_log()
        rc = lib.lbm_closure_relaxation(p(params), p(params), p(fields[0]), p(fields[1]),
                                        p(fields[2]), C.c_int64(nx), C.c_int64(ny), p(fields[3]),
                                        C.c_float(0.6), C.c_float(0.1), C.c_float(0.1), p(fields[0]),
                                        None)
        assert rc == 0, lib.lbm_last_error()
        assert lib.fake_take_log().decode().startswith(f"{device} ")


@pytest.mark.parametrize("steps", [20, 4000, 4002, 12000])
def test_calls_of_any_length_fall_back_to_single_steps(lib, steps):
    """Where a cooperative grid does not fit (a partition of the GPU), a call takes single steps,
    however many launches the resident kernel would have made of it, and so do later calls."""
    sim = FakeSim(lib, (256, 256))
    try:
        lib.fake_set_cooperative_limit(64)
        sim.check(sim.iterate(steps))
        assert set(sim.kernels()) == {"aa_step_kernel"}
    finally:
        lib.fake_set_cooperative_limit(-1)
    sim.check(sim.iterate(steps))
    assert set(sim.kernels()) <= {"aa_step_kernel"}
    sim.close()


def test_a_failure_after_the_first_launch_is_an_error(lib):
    sim = FakeSim(lib, (64, 64))
    lib.fake_fail_launch(1, 720)  # cudaErrorCooperativeLaunchTooLarge at the second launch
    assert sim.iterate(8000) != 0
    assert sim.kernels() == ["aa_resident_kernel"]
    sim.check(sim.iterate(8000))
    assert sim.kernels() == ["aa_resident_kernel"] * 2
    sim.close()


@pytest.mark.parametrize("counts,steps", [((64, 64), 8000), ((64, 64), 2), ((30, 20, 10), 4),
                                          ((64, 64, 256), 4)])
def test_a_failed_launch_is_reported_once(lib, counts, steps):
    """The error of a launch that fails is that call's; the next call does not meet it again."""
    sim = FakeSim(lib, counts)
    lib.fake_fail_launch(1, 701)  # cudaErrorLaunchOutOfResources at the second launch
    assert sim.iterate(steps) != 0
    sim.check(lib.lbm_equilibrate(sim.h))
    sim.check(sim.iterate(2))
    sim.close()


def test_a_poll_limit_does_not_change_the_kernel(lib):
    sim = FakeSim(lib, (64, 64))
    for polls in (0, 1 << 20, -1):
        sim.check(lib.lbm_set_spin_limit(sim.h, C.c_int64(polls)))
        sim.check(sim.iterate(20))
        assert sim.kernels() == ["aa_resident_kernel"]
    sim.close()


@pytest.mark.parametrize("counts,storage,kind,tracer,staged", [
    # 3D in 16 bits, rows of several tiles and of one.
    ((32, 48, 512), "f16", 1, "", False), ((70, 90, 512), "f16", 1, "", True),
    ((32, 48, 1024), "f16", 0, "", False), ((70, 45, 1024), "bf16", 0, "", True),
    ((128, 100, 512), "f16", 1, "32", False), ((128, 100, 512), "f16", 0, "32", False),
    ((32, 48, 512), "f16", 0, "16", False), ((40, 90, 768), "bf16", 0, "16", True),
    ((40, 90, 768), "f16", 1, "16", False),
    ((24, 48, 256), "f16", 1, "", False), ((64, 64, 256), "f16", 1, "", True),
    ((48, 64, 256), "f16", 0, "32", False), ((64, 64, 256), "f16", 0, "32", True),
    ((64, 64, 256), "f16", 1, "32", False), ((64, 90, 256), "f16", 1, "32", True),
    ((64, 64, 256), "f16", 0, "16", True), ((64, 90, 256), "f16", 1, "16", False),
    ((100, 100, 256), "f16", 1, "16", True),
    # 3D in full precision.
    ((24, 48, 256), "f32", 0, "", False), ((48, 64, 256), "f32", 0, "", True),
    ((128, 128, 256), "f32", 1, "", False), ((128, 64, 512), "f32", 0, "", False),
    ((128, 128, 256), "f32", 0, "32", False), ((100, 100, 256), "f64", 0, "", False),
    # 2D.
    ((4096, 2048), "f16", 1, "", False), ((2048, 512), "f16", 0, "32", False),
    ((1500, 1536), "f16", 0, "32", True), ((1500, 1536), "f16", 1, "16", False),
    ((1500, 2560), "f16", 1, "16", True), ((1500, 2560), "bf16", 0, "16", True),
    ((4096, 2048), "f32", 0, "", False), ((4096, 2048), "f32", 1, "32", True),
    ((2048, 1024), "f32", 1, "32", False), ((1500, 2560), "f64", 0, "", False),
])
def test_staged_where_it_is_the_faster_kernel(lib, counts, storage, kind, tracer, staged):
    """One domain on each side of every line of staged_pays (aa_launch.cuh)."""
    sim = FakeSim(lib, counts, kind=kind, storage=storage, tracer=tracer)
    sim.check(sim.iterate(2))
    kernels = set(sim.kernels())
    assert kernels == {"aa_tma_kernel"} if staged else "aa_tma_kernel" not in kernels
    sim.close()


def test_small_simulations_side_by_side_do_not_queue_for_the_chip(lib):
    """Resident launches that would take three turns or more give way to single steps, which overlap,
    while the simulations before them have not been waited for."""

    def kernels(counts, together):
        sims = [FakeSim(lib, counts) for _ in range(together)]
        out = []
        for s in sims:
            s.check(s.iterate(14))
            out.append(set(s.kernels()))
        # A simulation that has been waited for does not count: one of them alone, in turn.
        for s in sims:
            s.check(lib.lbm_synchronize(s.h))
        for s in sims:
            s.check(s.iterate(14))
            assert set(s.kernels()) == {"aa_resident_kernel"}
            s.check(lib.lbm_synchronize(s.h))
        for s in sims:
            s.close()
        return [k == {"aa_resident_kernel"} for k in out]

    assert kernels((128, 128), 4) == [True, True, False, False]
    assert kernels((64, 64), 6) == [True] * 4 + [False] * 2  # 64 of 148 CTAs each
    assert kernels((600, 400), 4) == [True] * 4  # large enough to be faster in turns
    assert kernels((12, 13), 20) == [True] * 20  # a few CTAs each


@pytest.mark.parametrize("counts,storage,steps,launches", [
    ((64, 64), "f32", 8004, [0, 0, 0, 3]), ((64, 64), "f32", 2, [2, 0, 0, 0]),
    ((500, 410), "f16", 6, [0, 6, 0, 0]), ((50, 40, 30), "f32", 30, [30, 0, 0, 0]),
    ((64, 64, 256), "f16", 30, [0, 0, 30, 0])])
def test_launches_are_counted_by_kernel(lib, counts, storage, steps, launches):
    sim = FakeSim(lib, counts, storage=storage)
    sim.check(sim.iterate(steps))
    got = (C.c_int64 * 4)()
    sim.check(lib.lbm_kernel_launches(sim.h, got, 4))
    assert list(got) == launches
    direct, staged = C.c_int64(), C.c_int64()
    sim.check(lib.lbm_launch_counts(sim.h, C.byref(direct), C.byref(staged)))
    assert (direct.value, staged.value) == ((0, steps) if launches[2] else (steps, 0))
    assert lib.lbm_kernel_launches(sim.h, got, 3) != 0 and lib.lbm_kernel_launches(sim.h, None, 4) != 0
    sim.close()


@pytest.mark.parametrize("counts,storage,kernel", [
    ([(400, 505)] * 10, "f32", "flat"), ([(500, 505)] * 10, "f32", "rows"),
    ([(500, 512)] * 16, "f16", "flat"), ([(500, 512)] * 20, "bf16", "rows"),
    ([(300, 100)] * 85, "f32", "flat"), ([(300, 100)] * 88, "f32", "rows"),
    ([(100, 256)] * 100, "f32", "flat"), ([(100, 257)] * 100, "f32", "rows"),
    ([(100, 600)] * 43, "f32", "flat"), ([(100, 600)] * 44, "f32", "step"),
    ([(64, 512), (256, 64)], "f32", "flat")])
def test_flat_ensembles(lib, counts, storage, kernel):
    """The default kernel on each side of the flat kernel's lines, and the Python class's copy of them."""
    from boltzmann_b200.ensemble import takes_flat

    h, om = C.c_void_p(), (C.c_float * len(counts))(*[1.5] * len(counts))
    arr = (C.c_int64 * (2 * len(counts)))(*[c for pair in counts for c in pair])
    assert lib.lbm_ensemble_create(len(counts), arr, 0, om, om, STORAGE[storage], C.byref(h)) == 0
    lib.fake_take_log()
    assert lib.lbm_ensemble_iterate(h, C.c_int64(2), 0) == 0, lib.lbm_last_error()
    assert f"ensemble_{kernel}_kernel" in lib.fake_take_log().decode()
    assert takes_flat(counts, storage) == (kernel == "flat")
    lib.lbm_ensemble_destroy(h)


@pytest.mark.parametrize("counts,storage,steps,kernel", [
    ((64, 64), "f32", 4, "aa_step_kernel"), ((64, 64), "f32", 6, "aa_resident_kernel"),
    ((500, 400), "f32", 12, "aa_resident_kernel"), ((500, 400), "f32", 10, "aa_step_kernel"),
    ((280, 280), "f64", 10, "aa_resident_kernel"), ((290, 290), "f64", 10, "aa_step_kernel"),
    ((499, 400), "f16", 2, "aa_step_kernel"), ((501, 400), "f16", 2, "aa_step2_kernel"),
    ((60, 160, 72), "f16", 2, "aa_step_kernel"), ((61, 160, 72), "bf16", 2, "aa_step2_kernel"),
    ((501, 400), "f32", 2, "aa_step_kernel")])
def test_kernels_on_each_side_of_their_lines(lib, counts, storage, steps, kernel):
    sim = FakeSim(lib, counts, storage=storage)
    sim.check(sim.iterate(steps))
    assert set(sim.kernels()) == {kernel}
    sim.close()


@pytest.mark.parametrize("counts,storage,tracers,dependent", [
    ((30, 20, 10), "f32", 0, True), ((60, 50, 40), "f32", 0, True), ((60, 50, 40), "f64", 0, True),
    ((16, 16, 16), "f64", 1, True), ((18, 18, 18), "f64", 1, False), ((23, 23, 23), "f32", 2, False),
    ((40, 30, 30), "f32", 2, True), ((200, 20), "f32", 3, True)])
def test_dependent_launches(lib, counts, storage, tracers, dependent):
    """Cells of much work (FP64, several tracers) are not launched as dependents where the grid fills
    half to three quarters of the chip's slots: here one CTA an SM, 148."""
    sim = FakeSim(lib, counts, storage=storage, tracer="32" if tracers else None)
    for _ in range(tracers - 1):
        sim.check(lib.lbm_add_tracer(sim.h, {2: 5, 3: 7}[len(counts)], 0, C.c_float(1.5), C.c_float(0),
                                     C.byref(C.c_int())))
    lib.fake_take_log()
    sim.check(sim.iterate(2))
    assert [name.endswith("+dependent") for _, name in sim.launched()] == [dependent] * 2
    sim.close()
