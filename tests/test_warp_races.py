"""The cooperative kernels' device code on the CPU, one thread per lane, under
ThreadSanitizer (warp_threads/warp_threads.h): lanes that share the slot array are ordered
by __syncwarp alone, so an access that relies on the warp's lanes staying together is
reported, whatever order they ran in; and the results equal the CPU oracle's bit for bit."""
import os
import re
import subprocess

import numpy as np
import pytest

HERE = os.path.join(os.path.dirname(os.path.abspath(__file__)), "warp_threads")
CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "warp_reactor_gb300", "csrc")
INCLUDE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "include")

# the PTX accesses of wr_coop.cuh, in C++
PTX = {
    'asm volatile("ld.shared.b64 %0, [%1];" : "=l"(v) : "r"(addr));': "v = slots[addr / 8];",
    'asm volatile("st.shared.b64 [%0], %1;" ::"r"(addr), "l"(v) : "memory");': "warp::store(slots, addr, v);",
    'asm volatile("ld.global.nc.v2.u64 {%0, %1}, [%2];" : "=l"(v.x), "=l"(v.y) : "l"(p));': "v = *p;",
    'asm volatile("ld.global.nc.u64 %0, [%1];" : "=l"(v) : "l"(p));': "v = *p;",
}


def compile_program(tmp, name, parts):
    """``name``.cpp with the device code ``parts`` as device_code.h, under the sanitizer."""
    for header in ("wr_coop.cuh", "wr_kernels.cuh", "wr_physics.cuh", "wr_math.h", "wr_diff.cuh",
                   "wr_coop_cta32.cuh"):
        src = open(os.path.join(CSRC, header)).read().replace('"../../include/', f'"{INCLUDE}/')
        if header == "wr_coop.cuh":
            for asm, cxx in PTX.items():
                assert src.count(asm) == 1, asm
                src = src.replace(asm, cxx)
            assert "asm" not in src
        if header == "wr_math.h":
            host = "#else\n    return a / b;\n#endif"
            assert src.count(host) == 1
            src = src.replace(host, host.replace("a / b", "native_division(a, b)"))
        # shared by the block, once: its dynamic shared memory is the program's array sm
        src = re.sub(r"(?<!extern )__shared__ ", "static ", src)
        (tmp / header).write_text(src)
    (tmp / "cuda_runtime.h").write_text("#pragma once\nusing cudaError_t = int;\nusing cudaStream_t = void*;\n")
    (tmp / "cooperative_groups.h").write_text(
        "#pragma once\nnamespace cooperative_groups {\nstruct cluster_group {\n    void sync() {}\n"
        "    template <class T>\n    T* map_shared_rank(T* p, int) { return p; }\n};\n"
        "inline cluster_group this_cluster() { return {}; }\n}\n")
    (tmp / "device_code.h").write_text(parts)
    exe = str(tmp / name)
    r = subprocess.run(["g++", "-std=c++20", "-O1", "-g", "-fsanitize=thread", "-ffp-contract=off", "-Wno-unknown-pragmas",
                        "-I", str(tmp), "-I", HERE, "-I", CSRC, os.path.join(HERE, name + ".cpp"), "-o", exe, "-pthread"],
                       capture_output=True, text=True)
    if "tsan" in r.stderr and "cannot find" in r.stderr:
        pytest.skip("no ThreadSanitizer runtime here")
    assert r.returncode == 0, r.stderr[-4000:]
    return exe


def run_program(exe, *args):
    r = subprocess.run([exe, *map(str, args)], capture_output=True, text=True, timeout=600,
                       env={**os.environ, "TSAN_OPTIONS": "halt_on_error=0 exitcode=66"})
    if "unexpected memory mapping" in r.stderr:
        pytest.skip("ThreadSanitizer cannot map its shadow here")
    races = sorted(set(re.findall(r"SUMMARY: ThreadSanitizer: data race (.*)", r.stderr)))
    assert not races, "\n".join(races[:20])
    assert r.returncode == 0, r.stderr[-2000:]
    return r.stdout


def advance_tables(G):
    """The tables of G lanes per cell as wr_adv_coop.cuh presents them to the kernels."""
    unit = open(os.path.join(CSRC, "wr_adv_coop.cuh")).read()
    tables = unit[unit.index("namespace cp ="):unit.index("static_assert(coop::kRes")].replace(
        "WR_CAT(coop, WR_COOP_G)", f"coop{G}").replace("int first(int w) { ", "int first(int w) { started(w); ")
    assert "started" in tables
    return f'#include "generated/coop_prog_g{G}.h"\n#include "wr_coop.cuh"\nnamespace wr {{\n{tables}\n}}\n'


@pytest.fixture(scope="module", params=[8, 16, 32])
def advance(request, built, tmp_path_factory):
    parts = advance_tables(request.param)
    return compile_program(tmp_path_factory.mktemp(f"advance{request.param}"), "advance", parts)


def burn(advance, tmp, oracle, wr, cells, dt):
    rec = np.zeros((len(cells), 16))
    rec[:, :14], rec[:, 14], rec[:, 15] = cells["xn"], cells["T"], dt
    (tmp / "in").write_bytes(rec.tobytes())
    programs = [int(w) for w in run_program(advance, tmp / "in", tmp / "out").split()]
    got = np.frombuffer((tmp / "out").read_bytes()).reshape(-1, 23)
    want = cells.copy()
    for i in range(len(cells)):
        assert oracle.burn(want[i:i + 1], np.broadcast_to(dt, len(cells))[i]) == wr.SUCCESS
    for i, name in enumerate(("internal_steps", "rhs_calls", "jacobian_calls", "decompositions", "linear_solves",
                              "accepted_steps", "rejected_steps")):
        assert (got[:, 15 + i] == want["stats"][name]).all(), name
    assert got[:, :14].tobytes() == want["xn"].tobytes()
    assert got[:, 14].tobytes() == want["e"].tobytes() and (got[:, 22] == wr.SUCCESS).all()
    return want["stats"], programs


def test_advance(advance, tmp_path, oracle_port, wr):
    """Cells with accepted and rejected attempts: alone in the warp, in pairs, one left over."""
    cells = wr.make_batch_grid(3, 3)
    stats, _ = burn(advance, tmp_path, oracle_port, wr, cells, 1e13)
    assert stats["internal_steps"].sum() > stats["accepted_steps"].sum()


@pytest.mark.parametrize("order", [(0, 1), (1, 0)])
def test_group_without_cell_follows(advance, tmp_path, oracle_port, wr, order):
    """A cell that retries beside a group whose own cell is done: the group without a cell
    computes the other's attempts, so the warp's programs are those of the cell alone but
    for one Jacobian at the new company (at one cell per warp, of the cell alone)."""
    cells = wr.make_batch_grid(3, 2)
    cells[1]["xn"] *= 1e12  # dense and hot: stages from its rates are far from the cold cell's state
    both = [cells[list(order)], np.array([1e14, 1e-5])[list(order)]]  # five attempts (two rejected) and one
    stats, programs = burn(advance, tmp_path, oracle_port, wr, *both)
    assert (stats["internal_steps"] == np.array([5, 1])[list(order)]).all()
    _, alone = burn(advance, tmp_path, oracle_port, wr, cells[:1], 1e14)
    if len(programs) >= len(alone) + 3:  # one after the other
        want = alone + programs[len(alone):] if order == (0, 1) else programs[:-len(alone)] + alone
    else:
        want = programs[:3] + alone[:1] + alone[3:]
    assert programs == want


@pytest.fixture(scope="module")
def tiles(built, tmp_path_factory):
    parts = "inline void started(int) {}\n" + advance_tables(16) + '#include "wr_coop_cta32.cuh"\n'
    return compile_program(tmp_path_factory.mktemp("tiles"), "tiles", parts)


def test_tiles(tiles, tmp_path, oracle_port, wr):
    """The structured policy's block: 16 warps, a full tile and a ragged one after it, whose
    trials one warp decides; some warps of the second hold one cell, most none."""
    cells = np.tile(wr.make_batch_grid(1, 35, log10_tmin=2.5, log10_tmax=3.2)[32:], 12)[:35]  # few trials
    want = cells.copy()
    rc, dt = oracle_port.prepare(cells.copy(), 0, 0.0, 0, True)
    assert rc == wr.SUCCESS
    rc, cgs = oracle_port.run_cta32(want, perturb=True, max_steps=1)
    assert (rc, cgs) == (wr.SUCCESS, 1)
    assert want["stats"]["internal_steps"].sum() > want["stats"]["accepted_steps"].sum()  # rejected trials
    (tmp_path / "in").write_bytes(cells.tobytes())
    out = run_program(tiles, dt, tmp_path / "in", tmp_path / "out")
    assert [int(v) for v in out.split()] == [wr.SUCCESS, len(cells)]
    assert (tmp_path / "out").read_bytes() == want.tobytes()


@pytest.fixture(scope="module")
def controller(tmp_path_factory):
    return compile_program(tmp_path_factory.mktemp("controller"), "controller", "")


@pytest.mark.parametrize("err,erracc,hacc,h", [(0.3, 1.0, 0.0, 1e11), (40.0, 1.0, 0.0, 1e13), (1e-7, 1.0, 0.0, 3e5),
                                               (0.7, 1e-2, 2e10, 3e10), (2.5, 0.4, 1e9, 4e9)])
def test_controller(controller, oracle_port, err, erracc, hacc, h):
    """Both step sizes of the reference's controller (reproducer.cpp:7308-7327), in every
    lane; the first attempts of a burn (no accepted step yet) divide on the integer path."""
    out = run_program(controller, err, erracc, hacc, h).split()
    sizes = np.array([float.fromhex(v) for v in out[:-1]]).reshape(-1, 2)
    fac = max(1 / 6.0, min(1 / 0.2, oracle_port.cbrt(err) / 0.9))
    assert (sizes[:, 0] == h / fac).all()
    if hacc != 0.0:
        gus = max(1 / 6.0, min(1 / 0.2, hacc / h * oracle_port.cbrt(err * err / erracc) / 0.9))
        assert (sizes[:, 1] == h / max(fac, gus)).all()
    assert int(out[-1]) == 0


@pytest.fixture(scope="module")
def gradient(built, tmp_path_factory):
    unit = open(os.path.join(CSRC, "wr_diff_coop.cu")).read()
    device = unit[:unit.index("template <class KernelT>")] + "}  // namespace\n}  // namespace diff\n}  // namespace wr\n"
    assert device.count("int first(int w) { ") == 1
    device = device.replace("int first(int w) { ", "int first(int w) { program = w; ")
    return compile_program(tmp_path_factory.mktemp("gradient"), "gradient", device)


def run_map(gradient, mode, tmp, oracle, cells, dts, log_mult, qbar):
    mult = np.array([oracle.exp(p) for p in log_mult])
    (tmp / "in").write_bytes(np.array([len(cells), len(dts)], np.int32).tobytes() + dts.tobytes() + mult.tobytes() +
                             cells.tobytes() + qbar.tobytes())
    run_program(gradient, mode, tmp / "in", tmp / "out")
    out = np.frombuffer((tmp / "out").read_bytes()).reshape(len(cells), -1)
    return out[:, :15], out[:, 15:30], out[:, 30:] * mult


def test_forward_map(gradient, tmp_path, oracle_port, wr):
    """Two cells one after the other in the warp, with rejected attempts: the oracle's final
    states, bit for bit."""
    from oracle import oracle as O
    cells, dts = wr.make_batch_grid(3, 3)[1:], np.array([1e13, 2e13])
    log_mult = np.random.default_rng(1).normal(0, 0.01, O.load_diff().num_multipliers)
    rc, want, _, counts = O.load_diff().record(cells, dts, perturb=False, log_mult=log_mult)
    assert rc == wr.SUCCESS
    q, _, _ = run_map(gradient, "forward", tmp_path, oracle_port, cells, dts, log_mult, np.zeros((2, 15)))
    assert q.tobytes() == want.tobytes()


def test_adjoint(gradient, tmp_path, oracle_port, wr):
    """The adjoint of the same map.  Its programs' slot array is larger than the forward
    programs', and none of them may store into the slot that is the smaller array's sink
    but to keep a value there.  Inner products with the tangent, <qbar, dq> = <ubar, du> +
    <pbar, dp>, to 1e-8 of their terms as on the GPU, for the electrons, H, H2 and T (the
    deuterium species, which start at 1e-40, end as rounding noise of the others)."""
    from oracle import oracle as O
    D, rng = O.load_diff(), np.random.default_rng(2)
    cells, dts = wr.make_batch_grid(3, 3)[1:], np.array([1e13, 2e13])
    log_mult = np.random.default_rng(1).normal(0, 0.01, D.num_multipliers)
    rc, q, hbuf, counts = D.record(cells, dts, perturb=False, log_mult=log_mult)
    assert rc == wr.SUCCESS
    qbar = np.zeros((len(cells), 15))
    for k in (0, 2, 8, 14):
        qbar[:, k] = rng.normal(size=len(cells)) / q[:, k]
    _, ubar, pbar = run_map(gradient, "adjoint", tmp_path, oracle_port, cells, dts, log_mult, qbar)
    du = rng.normal(size=(len(cells), 15)) * np.concatenate([cells["xn"], cells["T"][:, None]], axis=1)
    dp = rng.normal(size=D.num_multipliers)
    rc, _, dq = D.tangent(cells, dts, hbuf, counts, du=du, dlog_mult=dp, perturb=False, log_mult=log_mult)
    assert rc == wr.SUCCESS
    terms = np.concatenate([ubar * du, pbar * dp], axis=1)
    assert (np.abs((qbar * dq).sum(axis=1) - terms.sum(axis=1)) <= 1e-8 * np.abs(terms).sum(axis=1)).all()
