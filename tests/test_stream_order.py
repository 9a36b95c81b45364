"""Which of a step's operations are ordered after which, checked on the CPU.

The library runs with the CUDA runtime and cuFFT replaced by a stand-in
(host/stream_log.c) that records launches, copies, events and waits and runs no
kernel.  From the record each operation gets a vector clock over streams and the
host, so "a is ordered before b" is a comparison, whatever a GPU's timing would
have made of it."""
import os
import subprocess
import sys

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


@pytest.fixture(scope="session")
def standin(tmp_path_factory):
    so = tmp_path_factory.mktemp("standin") / "libstream_log.so"
    subprocess.run(["gcc", "-O1", "-w", "-shared", "-fPIC", "-o", str(so), os.path.join(HERE, "host", "stream_log.c")],
                   check=True)
    return so


class Ops:
    """The recorded operations with their vector clocks."""

    def __init__(self, log):
        clock, events, host = {}, {}, {}
        self.ops = []

        def join(a, b):
            for k, v in b.items():
                a[k] = max(a.get(k, 0), v)

        for line in log.splitlines():
            kind, s, x, name = line.split(" ", 3)
            c = clock.setdefault(s, {})
            if kind == "op":
                join(c, host)
                c[s] = c.get(s, 0) + 1
                self.ops.append((name, s, c[s], dict(c)))
            elif kind == "record":
                events[x] = dict(c)
            elif kind == "wait":
                join(c, events.get(x, {}))
            elif kind == "hostwait":
                join(host, events.get(x, {}))
            elif kind == "sync":
                join(host, c)
            elif kind == "syncall":
                for k in clock.values():
                    join(host, k)

    def find(self, name):
        return [o for o in self.ops if name in o[0]]

    @staticmethod
    def before(a, b):
        return b[3].get(a[1], 0) >= a[2]


def run(standin, tmp_path, lib, script, **env):
    log = tmp_path / "log"
    env = dict(os.environ, LD_PRELOAD=str(standin), STREAM_LOG=str(log), PYTHONPATH=ROOT, **env)
    r = subprocess.run([sys.executable, "-c", script], env=env, cwd=ROOT, capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stderr
    return Ops(log.read_text())


BATCH = """
from cafproject_gb300 import batch as B
from cafproject_gb300.cube import CubeError
b = B.Batch([(B.box_params(32, pp_on=%r), 1)], z_init=19.0, mode=B.GRAPH)
b.set_schedule(0.0, 4)
try:
    b.step(1)  # captures both parities; no kernel ran, so the check of the step's results fails
except CubeError as e:
    assert "box 0 step 1: " in str(e), e
"""


@pytest.mark.parametrize("pp_on", [True, False])
def test_captured_sums_before_the_codes_change(standin, tmp_path, built_lib, pp_on):
    """The captured step's velocity sums read the codes that the PP kick (in
    place) and the kicks after it rewrite: none may start before they are done."""
    o = run(standin, tmp_path, built_lib, BATCH % pp_on)
    sums = o.find("k_sigma")
    assert len(sums) == 2  # one per parity
    after = [k for k in o.find("k_pp_kick") + o.find("k_kick")]
    assert len(o.find("k_pp_kick")) == (2 if pp_on else 0) and len(o.find("k_kick")) == 6
    for i, s in enumerate(sums):
        end = sums[i + 1] if i + 1 < len(sums) else None
        seq = o.ops[o.ops.index(s):o.ops.index(end) if end else None]
        writers = [k for k in seq if k in after]
        assert writers
        for k in writers:
            assert o.before(s, k), k[0]


FAILED_KICK = """
from cafproject_gb300 import cube as C
from cafproject_gb300 import batch as B
p = B.box_params(32, pp_on=%r)
g = C.CubeGPU(p)
g.ic_zeldovich(19.0, seed=1)
g.set_sigma(g.get_sigma()[0], 0.0)  # what a re-sort of particles at rest leaves
try:
    (g.pp_particle_mesh if p.pp_on else g.particle_mesh)(0.4, 0.02)
    raise SystemExit("a zero sigma went through")
except C.CubeError as e:
    assert "sigma_vi must be positive" in str(e), e
g.get_field(C.FIELD_RHO_C)
"""


@pytest.mark.parametrize("pp_on", [True, False])
def test_failed_step_leaves_nothing_beside(standin, tmp_path, built_lib, pp_on):
    """A fused step that ends in an error while the coarse forces run beside it:
    whatever the next call does on the context's stream comes after them."""
    o = run(standin, tmp_path, built_lib, FAILED_KICK % pp_on)
    main = o.find("k_ic_gather")[0][1]
    read = o.find("memcpy2D")[-1]
    assert read[1] == main and o.ops[-1] == read
    beside = [k for k in o.ops if k[1] != main]
    assert any("k_deposit" in k[0] for k in beside) and any("c2r" in k[0] for k in beside)
    for k in beside:
        assert o.before(k, read), k[0]


OWN_FORCES = """
from cafproject_gb300 import cube as C
from cafproject_gb300 import batch as B
p = B.box_params(32, pp_on=False)
g = C.CubeGPU(p)
g.ic_zeldovich(19.0, seed=1)
g.%s_forces()
g.set_field(C.FIELD_FORCE_%s, g.get_field(C.FIELD_FORCE_%s))
for _ in range(2):
    g.%s_kick(0.4, 0.02)
"""


@pytest.mark.parametrize("level", ["fine", "coarse"])
def test_written_forces_keep_the_fast_kick(standin, tmp_path, built_lib, level):
    """The kick's fast path needs the maximum of the force mesh: after the
    caller has written the mesh it is found once, before the first kick."""
    F = level[0].upper()
    o = run(standin, tmp_path, built_lib, OWN_FORCES % (level, F, F, level))
    names = [k[0] for k in o.ops if "k_f2max" in k[0] or "k_kick" in k[0] or k[0] == "memcpy2D"]
    tail = ["max" if "f2max" in n else "kick" for n in names[len(names) - 1 - names[::-1].index("memcpy2D"):]]
    assert tail[1:3] == ["max", "kick"] and tail.count("max") == 1 and tail.count("kick") >= 2


BRICKS = """
from cafproject_gb300 import cube as C
from cafproject_gb300 import batch as B
g = C.CubeGPU(B.box_params(32, pp_on=False))
g.ic_zeldovich(19.0, seed=1)
for shape in (None, 0, -1):
    if shape is not None:
        g.set_option(C.OPT_DEPOSIT_%s, shape)
    g.%s_density()
for shape in (-2, 4):
    try:
        g.set_option(C.OPT_DEPOSIT_%s, shape)
        raise SystemExit("shape %%d went through" %% shape)
    except C.CubeError:
        pass
"""


@pytest.mark.parametrize("level", ["fine", "coarse"])
def test_default_brick_can_be_chosen_again(standin, tmp_path, built_lib, level):
    o = run(standin, tmp_path, built_lib, BRICKS % (level.upper(), level, level.upper()))
    names = [k[0] for k in o.find("k_deposit")]
    assert len(names) == 3 and names[0] == names[2] != names[1]


@pytest.mark.parametrize("level,fewest", [("fine", (8, 4, 4)), ("coarse", (8, 8, 8))])
def test_default_brick_goes_by_multiprocessors(standin, tmp_path, built_lib, level, fewest):
    """The smallest bricks while the default ones are fewer than the device's
    multiprocessors, whatever their number."""
    bricks = 1
    for b in fewest:
        bricks *= 16 // b
    script = BRICKS % (level.upper(), level, level.upper())
    first = [run(standin, tmp_path, built_lib, script, STREAM_SMS=str(n)).find("k_deposit")[0][0]
             for n in (152, bricks + 1, bricks)]
    assert first[0] == first[1] != first[2]


OVERFULL = """
from cafproject_gb300 import cube as C
from cafproject_gb300 import batch as B
g = C.CubeGPU(B.box_params(32, pp_on=False))
g.ic_zeldovich(19.0, seed=1)
g.set_option(C.OPT_RANK_WALK, 2)
try:  # the stand-in's count of the new state is far above np_max
    g.update_x(1.0, 1.0, 0.1)
    raise SystemExit("an overfull state went through")
except C.CubeError as e:
    assert "np_max" in str(e), e
"""


def test_overfull_state_is_refused_before_its_order_is_written(standin, tmp_path, built_lib):
    o = run(standin, tmp_path, built_lib, OVERFULL)
    assert o.find("k_sort_keys") and not o.find("k_sort_place") and not o.find("k_sort_gather")
