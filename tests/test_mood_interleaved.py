"""Two host-driven steps of one solver in flight at once (two threads, each on its own
stream) decide their redos independently.  The library's stage is stood in for on the CPU:
it writes the status word of the control block it is given, as the kernel does; the second
call runs whole between the first one's last stage and its decision."""
import ctypes as C

import pytest
import torch

from zoomy_b200 import _lib as L
from zoomy_b200.fvm.solver import HyperbolicSolver
from zoomy_b200.fvm.solver2 import TABLEAU_SSPRK2, MarchSolver

CELLS = 6


class Backend:
    """Stage calls of one solver: flags a cell where the state's first depth is negative."""

    stage_b_from_q0 = True

    def __init__(self):
        self.after_stage = None     # called once after the next flagging stage
        self.masked = []            # first depth of every stage run with a first-order mask

    def stage(self, cfg, Qk, Q0, Qo, alpha, beta, dt, hinv, fo, tr, ws, wsb, ctrl, st):
        depth = C.cast(Qk, C.POINTER(C.c_double))[CELLS]
        C.memmove(Qo, Qk, 4 * CELLS * 8)
        troubled = depth < 0.0 and not fo
        if fo:
            self.masked.append(depth)
        if tr:
            C.memset(tr, 1 if troubled else 0, CELLS)
        if troubled:
            block = C.cast(ctrl, C.POINTER(L.ZbCtrl)).contents
            block.status |= L.ZB_ST_TROUBLED
        # the last stage of a call is the one with a mask output or a second state
        if Q0 and self.after_stage is not None:
            run, self.after_stage = self.after_stage, None
            run()
        return L.ZB_OK


def solver(cls):
    s = cls.__new__(cls)
    s.be, s.mood = Backend(), True
    s.cfg = L.ZbSwe2dCfg()
    s.cfg.order = 2
    s._cfg_o1 = s.cfg
    s.tableau = TABLEAU_SSPRK2
    s._ws, s._ws_bytes = torch.zeros(8, dtype=torch.uint8), 8
    s._ctrl = torch.zeros(L.CTRL_BYTES, dtype=torch.uint8)
    s._probe = torch.zeros_like(s._ctrl)
    s._probes, s._probe_blocks = [], []
    s._s = lambda: C.c_void_p(0)
    return s


def state(depth):
    Q = torch.ones(4, CELLS, dtype=torch.float64)
    Q[1] = depth
    return Q


@pytest.mark.parametrize("first,second", [(-1.0, 2.0), (2.0, -1.0), (-1.0, -3.0)])
def test_step(first, second):
    s = solver(HyperbolicSolver)
    s.be.after_stage = lambda: s.step(0.1, 0.0, state(second), None)
    s.step(0.1, 0.0, state(first), None)
    # a redo is two masked stages, of the troubled states only
    want = [d for d in (second, first) if d < 0.0 for _ in range(2)]
    assert s.be.masked == want
    assert L.ZbCtrl.from_buffer_copy(s._ctrl.numpy().tobytes()).status == L.ZB_ST_TROUBLED
    # the free blocks are zero, one for each call that ran at once, and serve the next calls
    blocks = {p.data_ptr() for p, _ in s._probes}
    assert len(blocks) == len(s._probes) == 2
    assert not any(p.any() for p, _ in s._probes)
    s.step(0.1, 0.0, state(2.0), None)
    assert {p.data_ptr() for p, _ in s._probes} == blocks


def test_a_block_waits_for_its_fill_on_another_stream(monkeypatch):
    s = solver(HyperbolicSolver)
    waits = []
    monkeypatch.setattr(torch.cuda, "synchronize", lambda device=None: waits.append(device))
    for stream, depth in ((0, -1.0), (0, 2.0), (8, 2.0), (0, -1.0), (8, 2.0), (8, -1.0), (0, 2.0)):
        s._s = lambda v=stream: C.c_void_p(v)
        s.step(0.1, 0.0, state(depth), None)
    # only a block that a troubled step zeroes on one stream and that another one takes
    assert len(waits) == 2
    assert len(s._probe_blocks) == 1


@pytest.mark.parametrize("first,second", [(-1.0, 2.0), (2.0, -1.0), (-1.0, -3.0)])
def test_stage_loop(first, second):
    s = solver(MarchSolver)
    seen = {}

    def other():
        seen["second"] = s.stage_loop(state(second), None, 0.1)[1]

    # the hook fires after the last stage (the first one with an interleaved call armed)
    calls = {"n": 0}
    stage = s.be.stage

    def counted(*a):
        calls["n"] += 1
        if calls["n"] == len(s.tableau):
            s.be.after_stage = other
        return stage(*a)

    s.be.stage = counted
    seen["first"] = s.stage_loop(state(first), None, 0.1)[1]
    assert seen == {"first": first < 0.0, "second": second < 0.0}
