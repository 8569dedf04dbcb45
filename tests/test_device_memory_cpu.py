"""Device memory as the host code keeps it, without a device: the library's
host sources over tests/cxx/fake_cuda.cpp, whose allocations are host memory
with every copy, fill and launch argument checked against them."""
import ctypes
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

from pannde_gb300 import _native as N
from pannde_gb300 import cases
from pannde_gb300.build import _cuda_home
from pannde_gb300.solver import Batch, Solver

ROOT = Path(__file__).resolve().parent.parent
CSRC = ROOT / "pannde_gb300" / "csrc"


@pytest.fixture(scope="module")
def fake_lib(tmp_path_factory):
    if not shutil.which("g++") or not (_cuda_home() / "include" / "cuda_runtime.h").exists():
        pytest.skip("no g++ or no CUDA headers")
    out = tmp_path_factory.mktemp("fake")
    inc = ["-I", str(_cuda_home() / "include"), "-I", str(CSRC), "-I", str(ROOT / "include")]
    srcs = [ROOT / "tests" / "cxx" / "fake_cuda.cpp"] + [CSRC / f"pn_{n}.cpp" for n in
            ("setup", "table", "grid", "capi", "batch", "energy", "partition")]
    jobs = [subprocess.Popen(["g++", "-std=c++17", "-O1", "-fPIC", "-fopenmp", *inc, "-c", str(s), "-o",
                              str(out / (s.stem + ".o"))], stderr=subprocess.PIPE, text=True) for s in srcs]
    for j in jobs:
        err = j.communicate()[1]
        assert j.returncode == 0, err
    so = out / "libfake.so"
    r = subprocess.run(["g++", "-shared", "-fopenmp", "-o", str(so)] + [str(out / (s.stem + ".o")) for s in srcs] +
                       ["-Wl,--no-undefined", "-Wl,-Bsymbolic"], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return so


@pytest.fixture
def fake(fake_lib, monkeypatch):
    lib = N.load(fake_lib)
    lib.fake_first_fault.restype = ctypes.c_char_p
    for f in ("fake_held", "fake_launches", "fake_chunk_choices", "fake_launches_without_reciprocals"):
        getattr(lib, f).restype = ctypes.c_int64
    lib.fake_set_room.argtypes = [ctypes.c_int64]
    monkeypatch.setattr(N, "_lib", lib)
    monkeypatch.delenv("PN_HBM_BUDGET_BYTES", raising=False)
    lib.fake_reset()
    yield lib
    assert lib.fake_faults() == 0, lib.fake_first_fault().decode()


def plate(**kw):
    return cases.al_plate_case(**dict(dict(nx=14, ny=11, nz=6, h=0.1e-3, nsteps=30, radius=0.5e-3, n_sensors=5), **kw))


@pytest.mark.parametrize("how", ["budget", "device"])
def test_launches_after_the_reciprocals_made_room(fake, monkeypatch, how):
    """Exact form: the first solve's signal table takes the room that the
    reciprocals held; that solve's launches, and the later ones, are given none."""
    c = plate()
    with Solver.from_case(c, "f64_exact") as s:
        s.solve(3)
        full, held = s.info()["device_bytes"], fake.fake_held()
    assert fake.fake_launches() == 6 and fake.fake_launches_without_reciprocals() == 0
    if how == "budget":
        monkeypatch.setenv("PN_HBM_BUDGET_BYTES", str(full - 1))
    else:
        fake.fake_set_room(held - 1)
    with Solver.from_case(c, "f64_exact") as s:
        s.solve(3)
        assert s.info()["device_bytes"] == full - 48 * (c.mesh.n_nodes + c.mesh.n_cells)
        assert fake.fake_launches_without_reciprocals() == 6
        s.solve(2)
    assert fake.fake_launches_without_reciprocals() == 10


@pytest.mark.parametrize("form, prec", [("grid", "f32"), ("grid", "f64"), ("table", "f64"), ("table", "f64_exact")])
@pytest.mark.parametrize("how", ["solve", "signals", "batch"])
def test_signal_rows_of_sources_added_later(fake, form, prec, how):
    """The signal table was sized for fewer sources: rows of more need a larger one."""
    if how == "batch" and prec == "f64_exact":
        pytest.skip("not batched")
    c = plate()
    more = [cases.WindowSource(N.PN_SOURCE_FORCE, g, d, c.sources[0].center, c.sources[0].radius, c.sources[0].ds,
                               c.sources[0].times, c.sources[0].values) for g in range(1, 5) for d in range(3)]
    with Solver.from_case(c, prec, form=form) as s, Batch() as b:
        s.solve(2)
        s.add_sources(more)
        if how == "solve":
            s.solve(2)
        elif how == "signals":
            s.solve_signals(np.zeros((1000, 13)))
        else:
            b.add(s)
            b.solve(2)
            b.solve_noalloc(2)


@pytest.mark.parametrize("n_sources", [1, 9])
@pytest.mark.parametrize("form", ["grid", "table"])
def test_caller_signals_leave_rows_for_the_allocation_free_batch(fake, form, n_sources):
    """A solver advanced by solve_signals alone is taken by solve_noalloc,
    whether its launches carry the values (few sources) or a table does."""
    c = plate()
    c.sources = [cases.WindowSource(N.PN_SOURCE_FORCE, g // 3, g % 3, c.sources[0].center, c.sources[0].radius,
                                    c.sources[0].ds, c.sources[0].times, c.sources[0].values)
                 for g in range(n_sources)]
    with Solver.from_case(c, "f32", form=form) as s, Batch() as b:
        s.solve_signals(np.zeros((3, n_sources)))
        b.add(s)
        held = fake.fake_held()
        b.solve_noalloc(7)
        assert fake.fake_held() == held or held + 262144 == fake.fake_held()  # (the fixed scratch, once)


@pytest.mark.parametrize("form, prec, block", [("grid", "f32", 512), ("grid", "f64", 520), ("grid", "df64", 520),
                                               ("table", "f32", 232), ("table", "f64", 240), ("table", "df64", 240)])
def test_members_the_fixed_scratch_takes(fake, form, prec, block):
    """A member's argument block keeps its size: the allocation-free batch
    solve takes as many members as its 256 KiB hold, and no more."""
    def room(n):
        starts = 2 * (n + 1) if form == "grid" else n + 1
        return 2 * (-(-block * n // 256) * 256) + 2 * (-(-starts * 4 // 256) * 256)
    most = max(n for n in range(1, 1000) if room(n) <= 256 * 1024)
    m = cases.voxel_mesh(np.ones((2, 2, 2), dtype=bool), 1e-4)
    c = cases.Case("tiny", m, np.array([2700.0]), cases.c21_from_6x6(cases.isotropic(70e9, 0.33))[None],
                   np.zeros(m.n_cells, np.int32), 1e-9)
    sv = [Solver(m, c, c.dt, prec, form) for _ in range(most + 1)]
    with Batch() as b:
        for s in sv[:most]:
            b.add(s)
        b.solve_noalloc(1)
        b.add(sv[most])
        with pytest.raises(N.PnError) as e:
            b.solve_noalloc(1)
        assert f"{most + 1} members need {room(most + 1)} bytes" in e.value.msg
    for s in sv:
        s.close()


def test_batch_calls_keep_the_chosen_chunk_length(fake):
    """A batch chooses its chunk length once per set of members and tile rows,
    not from every member's lattice in every call."""
    c = plate()
    with Solver.from_case(c, "f32", form="grid") as s, Solver.from_case(c, "f32", form="grid") as t, Batch() as b:
        b.add(s)
        b.solve(5)
        first = fake.fake_chunk_choices()
        for _ in range(3):
            b.solve(5)
        b.solve_noalloc(5)
        assert first > 0 and fake.fake_chunk_choices() == first
        b.add(t)
        b.solve(5)
        assert fake.fake_chunk_choices() == 2 * first


@pytest.mark.parametrize("form, prec", [("grid", "f64"), ("grid", "f32"), ("table", "f32"), ("table", "f64_exact")])
def test_device_bytes_are_what_is_held(fake, form, prec):
    """Sensors set again, sources added, a longer signal table: what was given
    back is not counted."""
    c = plate()
    with Solver.from_case(c, prec, form=form) as s:
        before = fake.fake_held() - s.info()["device_bytes"]
        s.solve(2)
        once = s.info()["device_bytes"]
        for _ in range(3):
            s.set_sensors(c.sensors, 30)
        assert s.info()["device_bytes"] == once
        s.add_sources([cases.WindowSource(N.PN_SOURCE_FORCE, 1, 0, c.sources[0].center, c.sources[0].radius,
                                          c.sources[0].ds, c.sources[0].times, c.sources[0].values)])
        s.solve(2)
        s.get_state()
        s.energy()
        assert fake.fake_held() - s.info()["device_bytes"] == before  # (what others hold)


@pytest.mark.parametrize("nx, ny", [(5, 4), (62, 4), (70, 40)])
def test_path_flags_take_no_more_than_three_words_a_tile(fake, monkeypatch, nx, ny):
    """The FP64 form's flags keep to the room that three words per tile took."""
    c = plate(nx=nx, ny=ny, radius=0.1e-3)
    got = {}
    for path in ("fp64", ""):  # (fp64: the form without flags)
        monkeypatch.setenv("PN_F64_PATH", path)
        with Solver.from_case(c, "f64", form="grid") as s:
            got[path] = s.info()["device_bytes"]
    tiles = (nx // 31 + 1) * (ny // 7 + 1)
    assert got[""] - got["fp64"] <= 16 + 12 * tiles  # 16: the path counts


@pytest.mark.parametrize("prec", ["f32", "f64"])
def test_slots_rows_give_way_to_a_budget(fake, monkeypatch, prec):
    """Grid form: what lies behind the slots' ranges takes no room that a
    budget does not have.  The least budget is that of the form without it (the
    classic kernel's, the tensor maps and tile tops beside it); up to the full
    size the solver holds no more than the budget, and its launches read live
    memory."""
    c = plate(nx=70, ny=30)

    def run(budget=None):
        if budget is None:
            monkeypatch.delenv("PN_HBM_BUDGET_BYTES", raising=False)
        else:
            monkeypatch.setenv("PN_HBM_BUDGET_BYTES", str(budget))
        others = fake.fake_held()
        with Solver.from_case(c, prec, form="grid") as s:
            s.solve(2)
            s.get_state()  # (staging and index maps)
            s.solve(2)
            assert budget is None or fake.fake_held() - others <= s.info()["device_bytes"] <= budget
            return s.info()["device_bytes"]

    full = run()
    monkeypatch.setenv("PN_GRID_KERNEL", "classic")
    classic = run()
    monkeypatch.delenv("PN_GRID_KERNEL")
    tiles = (70 // 31 + 1) * (30 // 7 + 1)
    flags = 16 + (4 * tiles + 7) // 8 * 8 + 24 if prec == "f64" else 0  # path counts, flags, column counts
    least = classic + 2 * 11 * 128 + 4 * tiles + flags
    assert least < full
    for budget in {full, full - 1, (full + least) // 2, least + 1, least}:
        run(budget)
    with pytest.raises(N.PnError) as e:
        run(least - 1)
    assert e.value.code == N.PN_ERR_ALLOC


def test_another_solver_takes_the_reciprocals_room(fake):
    """Device memory that holds one exact solver's reciprocals or another
    solver, not both: the other solver is created, and the first goes on
    without; one whose launches a stream capture recorded keeps them."""
    c = plate(nx=30, ny=30)
    base = fake.fake_held()
    with Solver.from_case(c, "f64_exact") as a:
        a.solve(2)
        one = fake.fake_held() - base
        recips = 48 * (c.mesh.n_nodes + c.mesh.n_cells)
        with Solver.from_case(c, "f32", form="table") as b:
            b.solve(2)
            two = fake.fake_held() - base - one
    for captured in (False, True):
        fake.fake_reset()
        with Solver.from_case(c, "f64_exact") as a:
            fake.fake_set_capturing(captured)
            a.solve(2)
            fake.fake_set_capturing(False)
            assert fake.fake_launches_without_reciprocals() == 0
            fake.fake_set_room(base + one + two - recips)
            if captured:
                with pytest.raises(N.PnError):
                    Solver.from_case(c, "f32", form="table").solve(2)
                a.solve(1)
                assert fake.fake_launches_without_reciprocals() == 0
                continue
            with Solver.from_case(c, "f32", form="table") as b:
                b.solve(2)
                a.solve(2)
                assert fake.fake_launches_without_reciprocals() == 4
                assert a.info()["device_bytes"] == one - recips


def test_reciprocals_leave_most_of_the_memory_free(fake):
    """They are taken only as a small part of what is free (other libraries
    cannot get them back), and a plan does not count them."""
    import ctypes as ct
    c = plate()
    base = fake.fake_held()
    recips = 48 * (c.mesh.n_nodes + c.mesh.n_cells)
    m, k1 = c.mesh.as_struct()
    tab, k2 = c.material_table()
    plan = N.PnPlan()
    N.check(fake.pn_plan_solver(ct.byref(m), None, ct.byref(tab), c.dt, N.PN_PREC_F64_EXACT, ct.byref(plan)))
    for room, without in ((plan.device_bytes + 9 * recips, False), (plan.device_bytes + 7 * recips, True)):
        fake.fake_reset()
        fake.fake_set_room(base + room)
        with Solver(c.mesh, c, c.dt, "f64_exact") as s:
            assert s.info()["device_bytes"] == plan.device_bytes + (0 if without else recips)
            s.solve(1)
            assert fake.fake_launches_without_reciprocals() == (2 if without else 0)


def test_table_bytes_are_of_what_the_solver_holds(fake, monkeypatch):
    c = plate()
    shuffled = np.random.default_rng(3).permutation(c.mesh.n_cells)
    many = cases.Case("m", cases.HexMesh(c.mesh.x, c.mesh.y, c.mesh.z, c.mesh.hexes[shuffled]), c.density, c.cij,
                      c.cell_material[shuffled], c.dt)

    def of(case, prec, form="table"):
        with Solver(case.mesh, case, case.dt, prec, form) as s:
            return s.table_bytes()
    assert of(c, "f32", "grid") == (0, 0)
    assert of(c, "f32") == (5, 5)  # a plate: patterns, one spacing
    assert of(many, "f64") == (32, 5)  # the nodes' cells in no order: a table
    assert of(c, "f64_exact") == (32 + 24 + 48, 32 + 24 + 48)
    fake.fake_set_room(fake.fake_held() + 3000000)
    assert of(plate(nx=40, ny=40), "f64_exact") == (32 + 24, 32 + 24)  # no reciprocals held


def test_a_batch_takes_the_reciprocals_room(fake):
    c = plate(nx=30, ny=30)
    with Solver.from_case(c, "f64_exact") as a, Solver.from_case(c, "f32", form="table") as s, Batch() as b:
        a.solve(1)
        s.solve(1)
        b.add(s)
        fake.fake_set_room(fake.fake_held() + 16)
        b.solve(2)  # its staging
        a.solve(1)
        assert fake.fake_launches_without_reciprocals() == 2
