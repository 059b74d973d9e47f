"""The plan of automata that are only aligned (fbw_b200_prepare_alignment) is the plan of fbw_b200_prepare without the
notes for the sweeps, and it is the one that fast_viterbi builds: one launch fewer where the general builder takes the
batch, with the same alignment."""
import ctypes

import numpy as np
import pytest
import torch

from test_automaton_sizes_gpu import batch, on_device
from test_zz_no_alloc import LIB

pytestmark = pytest.mark.gpu

FIELDS = 14 + 3 + 3 * 8 + 3  # of fbw_b200_summary before `reserved`


# 4 sequences; an average above 2048 edges goes to the general builder, below it only a sequence above 4096 does
@pytest.mark.parametrize("S,deg,general", [(60, 3, False), (1800, 4, True), (1500, 3, True)])
def test_plan_of_an_alignment(cuda, S, deg, general):
    import i6_native_ops_b200.fast_viterbi as m

    lib = ctypes.CDLL(LIB)
    i64, vp = ctypes.c_int64, ctypes.c_void_p
    lib.fbw_b200_plan_bytes.restype = lib.fbw_b200_viterbi_bytes.restype = ctypes.c_size_t
    lib.fbw_b200_launch_count.restype = i64
    T, F = 60, 90
    e, w, se, lens, n, rng = batch(S, deg, T, F)
    E, B = e.shape[1], 4
    per = np.bincount(e[3], minlength=B)
    takes_general = per.max() > 4096 or E // B > 2048
    assert takes_general == general and (E // B > 2048) == (S == 1800)
    am, e, w, se, lens = on_device(cuda, rng.normal(4.0, 3.0, (T, B, F)).astype(np.float32), np.ascontiguousarray(e), w, se, lens)
    plan = torch.empty(lib.fbw_b200_plan_bytes(i64(B), i64(E), i64(n)), dtype=torch.uint8, device=cuda)
    args = [vp(x.data_ptr()) for x in (e, w, se, lens)] + [i64(x) for x in (T, B, F, E, n)]
    stream = vp(torch.cuda.current_stream().cuda_stream)
    room = [vp(plan.data_ptr()), ctypes.c_size_t(plan.numel()), stream]

    def prepared(build, build_general):
        before, s = lib.fbw_b200_launch_count(), (i64 * (FIELDS + 1))()
        assert build() == 0
        rc = lib.fbw_b200_plan_summary(vp(plan.data_ptr()), s, stream)
        if rc == 6:
            assert build_general() == 0
            rc = lib.fbw_b200_plan_summary(vp(plan.data_ptr()), s, stream)
        assert rc == 0
        return list(s), lib.fbw_b200_launch_count() - before

    full, launches = prepared(lambda: lib.fbw_b200_prepare(*args, *room), lambda: lib.fbw_b200_prepare_general(*args, *room))
    slim, fewer = prepared(lambda: lib.fbw_b200_prepare_alignment(*args, 0, *room),
                           lambda: lib.fbw_b200_prepare_alignment(*args, 1, *room))
    assert slim[:FIELDS] == full[:FIELDS]
    assert launches - fewer == (1 if takes_general else 0)
    assert (full[FIELDS] >> 32 != 0) == takes_general and slim[FIELDS] >> 32 == 0

    s = (i64 * (FIELDS + 1))(*slim)
    bytes_ = lib.fbw_b200_viterbi_bytes(s)
    work = torch.empty(bytes_, dtype=torch.uint8, device=cuda)
    alignment = torch.empty((T, B), dtype=torch.int32, device=cuda)
    scores = torch.empty(B, device=cuda)
    before = lib.fbw_b200_launch_count()
    assert lib.fbw_b200_viterbi(vp(plan.data_ptr()), s, vp(am.data_ptr()), vp(alignment.data_ptr()), vp(scores.data_ptr()), 0,
                                vp(work.data_ptr()), ctypes.c_size_t(bytes_), stream) == 0
    torch.cuda.synchronize()
    of_run = lib.fbw_b200_launch_count() - before
    before = lib.fbw_b200_launch_count()
    want = m.core.fast_viterbi(am, e, w, se, lens, n)
    assert lib.fbw_b200_launch_count() - before == fewer + of_run
    assert torch.equal(alignment, want[0]) and torch.equal(scores, want[1])
