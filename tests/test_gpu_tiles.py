"""The tile trajectory kernels against the oracle and against the row-block kernel: every tile count
with ragged and full sizes, one team per channel and one team for all channels (the same bits), the
packed route with and without whole zero tiles, and a density that is not Hermitian (the row-block
kernel)."""
import ctypes as C
import threading
import time

import numpy as np
import pytest

from oracle import fg_phi4_oracle as O

pytestmark = pytest.mark.gpu

WINDOW, NODES = 1.5, 8


def _state(d, z2, seed):
    from rcmps_b200 import objective
    from rcmps_b200.batch import random_state, z2_state
    r, k = (z2_state if z2 else random_state)(d, seed)
    return r, k, objective.stationary_state(O.left_canonical_q(r, k), r, tolerance=1e-13)[0]


def _batch(states, groups=0, symmetry=2):
    from rcmps_b200 import objective
    s = objective.settings_from_args(None, half_window=WINDOW, n_quad=NODES, kinetic_nodes=8, symmetry=symmetry,
                                     trajectory_groups=groups)
    R, K, rho = zip(*states)
    E, _, st, C, env = objective.fg_phi4_batch(R, K, rho, [1.0] * len(R), s, return_parts=True)
    return [(E[i], C[i], env[i], st[i]["accepted"], st[i]["rejected"]) for i in range(len(R))]


@pytest.mark.parametrize("d", [1, 2, 15, 16, 17, 32, 33, 48, 49, 64])
@pytest.mark.parametrize("z2", [False, True])
def test_quartic_against_the_oracle(gpu_context, d, z2):
    from rcmps_b200 import objective
    if z2 and d % 2:
        pytest.skip("Z2 states have an even D")
    r, k, rho = _state(d, z2, 60 + d)
    q = O.left_canonical_q(r, k)
    o = O.evaluate_quartic(r, q, rho, 1.0, half_window=WINDOW, n_quad=NODES, return_samples=True, packed_z2=z2)
    g = objective.evaluate_quartic_persistent_trajectory(r, q, rho, 1.0, half_window=WINDOW, n_quad=NODES,
                                                         return_samples=True, unpacked=not z2)
    assert (g["stats"]["accepted"], g["stats"]["rejected"]) == (o["stats"]["accepted"], o["stats"]["rejected"])
    assert abs(g["value"] - o["value"]) <= 1e-11 * max(abs(o["value"]), 1e-3)
    for out in (g, o):   # the library reports the scalar channel at the endpoint only
        out["samples"][:-1, -1] = 0
    for name in ("covector", "environment", "samples"):
        assert np.linalg.norm(g[name] - o[name]) <= 1e-11 * max(1.0, np.linalg.norm(o[name]))


def _quartic(ctx, states, symmetry=2, window=WINDOW):
    """The quartic part alone of a batch: per state the value, covector, environment and the
    controller's record."""
    import torch
    from rcmps_b200 import _lib, objective
    s = objective.settings_from_args(None, half_window=window, n_quad=NODES, symmetry=symmetry)
    n, dims = len(states), [len(x[0]) for x in states]
    dR, dK, dP = (objective._device(list(x)) for x in zip(*states))
    value = torch.zeros(n, dtype=torch.float64, device="cuda")
    cov = torch.zeros(sum(d * d for d in dims), dtype=torch.complex128, device="cuda")
    env = torch.zeros_like(cov)
    stats = (_lib.StateStats * n)()
    rc = ctx.lib.rcmps_quartic_batch(ctx.handle, n, (C.c_int * n)(*dims), (C.c_double * n)(*[1.0] * n), dR.data_ptr(),
                                     dK.data_ptr(), dP.data_ptr(), C.byref(s), value.data_ptr(), cov.data_ptr(),
                                     env.data_ptr(), stats, objective._stream())
    objective._raise_for(rc, ctx, stats[0], "quartic")
    cov, env = objective._unpack(cov, dims), objective._unpack(env, dims)
    return [(value[i].item(), cov[i], env[i], stats[i].as_dict()) for i in range(n)]


def _one_team_batch(ctx, states):
    """The states repeated until a launch takes one team per state: (copies, results)."""
    many = 8 * len(states)
    while many <= 2048:
        out = _quartic(ctx, [states[i % len(states)] for i in range(many)])
        if ctx.trajectory_layout(len(states[0][0])) == (1, many, 0):
            return many, out
        many *= 2
    raise AssertionError("no launch took one team per state")


@pytest.mark.parametrize("d,z2", [(80, False), (96, True), (100, False), (128, True)])
def test_large_tiles_against_the_row_blocks(gpu_context, d, z2):
    state = _state(d, z2, d)
    (e0, c0, v0, a0, r0), = _batch([state], groups=1)
    assert gpu_context.trajectory_layout(d) == (0, 0, 1)
    many, _ = _one_team_batch(gpu_context, [state])
    for n, teams in ((1, 7), (4, 7), (many, 1)):
        results = _batch([state] * n)
        assert gpu_context.trajectory_layout(d) == (teams, n, 0)
        for e, c, v, a, r in results:
            assert (a, r) == (a0, r0)
            assert abs(e - e0) <= 1e-12 * abs(e0)
            assert np.linalg.norm(c - c0) <= 1e-11 * np.linalg.norm(c0)
            assert np.linalg.norm(v - v0) <= 1e-11 * np.linalg.norm(v0)


@pytest.mark.parametrize("d", [9, 16, 24, 32, 40, 48, 50, 64, 80, 96, 100, 128])
def test_batch_and_lone_state_give_the_same_bits(gpu_context, d):
    states = [_state(d, i % 2 == 1 and d % 2 == 0, 10 * d + i) for i in range(3)]
    _, batch = _one_team_batch(gpu_context, states)
    for i, state in enumerate(states):
        value, cov, env, stats = _quartic(gpu_context, [state])[0]
        assert gpu_context.trajectory_layout(d) == (7, 1, 0)
        for b in batch[i::3]:
            assert b[0] == value
            assert np.array_equal(b[2], env)
            assert np.array_equal(b[1], cov)
            for name in ("attempts", "accepted", "rejected", "dense_steps", "t_end", "last_step", "min_step", "max_step",
                         "packed_z2"):
                assert b[3][name] == stats[name], name


@pytest.mark.parametrize("control", [dict(trajectory_groups=4), dict(precision=1)])
def test_kinetic_term_beside_row_blocks_is_the_one_alone(gpu_context, control):
    """Beside a trajectory on few CTAs the Gram-Schmidt steps keep their clusters, so the sums keep their
    order: the kinetic value in the call has the bits of the kinetic entry's."""
    import torch
    from rcmps_b200 import _lib, objective
    r, k, rho = _state(64, False, 4)
    s = objective.settings_from_args(None, half_window=WINDOW, n_quad=NODES, kinetic_nodes=64, symmetry=0, **control)
    _, _, stats = objective.fg_phi4_batch([r], [k], [rho], [1.0], s)
    value = torch.zeros(1, dtype=torch.float64, device="cuda")
    alone = (_lib.StateStats * 1)()
    dR, dK, dP = (objective._device([x]) for x in (r, k, rho))
    assert gpu_context.lib.rcmps_kinetic_batch(gpu_context.handle, 1, (C.c_int * 1)(64), dR.data_ptr(), dK.data_ptr(),
                                               dP.data_ptr(), C.byref(s), value.data_ptr(), None, None, alone,
                                               objective._stream()) == 0
    assert stats[0]["krylov_basis"] == alone[0].as_dict()["krylov_basis"]
    assert stats[0]["kinetic_value"] == value.item()
    assert stats[0]["krylov_residual"] == alone[0].krylov_residual


def test_density_that_is_not_hermitian_takes_the_general_equations(gpu_context):
    r, k, rho = _state(12, False, 3)
    bent = rho + 1e-9 * (r - r.conj().T)
    mixed = _batch([(r, k, rho), (r, k, bent)], symmetry=0)
    alone = [_batch([(r, k, rho)], symmetry=0)[0], _batch([(r, k, bent)], groups=1, symmetry=0)[0]]
    for got, want in zip(mixed, alone):
        assert got[3:] == want[3:]
        assert abs(got[0] - want[0]) <= 1e-13 * abs(want[0])
        assert np.linalg.norm(got[1] - want[1]) <= 1e-12 * np.linalg.norm(want[1])


@pytest.mark.parametrize("d,z2", [(12, False), (40, True)])
def test_the_layout_tells_which_kernel_ran(gpu_context, d, z2):
    state = _state(d, z2, 7)
    _batch([state])
    assert gpu_context.trajectory_layout(d) == (7, 1, 0)
    _batch([state], groups=2)
    assert gpu_context.trajectory_layout(d) == (0, 0, 1)
    r, k, rho = state
    bent = rho + 1e-9 * (r - r.conj().T)
    _batch([(r, k, bent)], symmetry=0)
    assert gpu_context.trajectory_layout(d) == (0, 0, 1)
    _batch([state] * 300)
    assert gpu_context.trajectory_layout(d) == (1, 300, 0)


def test_states_beside_one_that_is_not_hermitian(gpu_context):
    """Few states ride along in the row-block launch; more than it holds at once (it runs at most 16
    CTAs per SM) take their own, and keep their bits."""
    r, k, rho = _state(12, False, 3)
    bent = (r, k, rho + 1e-9 * (r - r.conj().T))
    want = _quartic(gpu_context, [(r, k, rho)], symmetry=0)[0]
    for few in (1, 30):
        got = _quartic(gpu_context, [bent] + [(r, k, rho)] * few, symmetry=0)
        assert gpu_context.trajectory_layout(12) == (0, 0, few + 1)
        for g in got[1:]:
            assert g[3]["accepted"] == want[3]["accepted"]
            assert abs(g[0] - want[0]) <= 1e-13 * abs(want[0])
            assert np.linalg.norm(g[1] - want[1]) <= 1e-12 * np.linalg.norm(want[1])
    many = 2400
    got = _quartic(gpu_context, [bent] + [(r, k, rho)] * many, symmetry=0)
    assert gpu_context.trajectory_layout(12) == (1, many, 1)
    for g in got[1::100]:
        assert g[0] == want[0] and np.array_equal(g[1], want[1]) and np.array_equal(g[2], want[2])
    alone = _quartic(gpu_context, [bent], symmetry=0)[0]
    assert abs(got[0][0] - alone[0]) <= 1e-13 * abs(alone[0])


@pytest.mark.parametrize("entry", [(0, 0), (3, 1), (1, 19), (19, 19)])
@pytest.mark.parametrize("bad", [complex(np.nan, 0.1), complex(0.1, np.nan), complex(np.inf, 0), complex(0, -np.inf)])
def test_a_density_that_is_not_finite_is_not_hermitian(gpu_context, entry, bad):
    """Through the C entry (the Python calls refuse it): the general equations, which stop at once."""
    from rcmps_b200 import objective
    r, k, rho = _state(20, False, 5)
    rho = rho.copy()
    rho[entry] = bad
    rho[entry[::-1]] = np.conj(bad)
    with pytest.raises(objective.DeviceControlFailure, match="nonfinite_error"):
        _quartic(gpu_context, [(r, k, rho)], symmetry=0)
    assert gpu_context.trajectory_layout(20) == (0, 0, 1)


def _in_threads(jobs):
    """The jobs side by side, a host thread and a stream each: their results and the wall time."""
    import torch
    out, start = [None] * len(jobs), threading.Barrier(len(jobs) + 1)

    def work(i):
        with torch.cuda.stream(torch.cuda.Stream()):
            start.wait()
            out[i] = jobs[i]()
    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(jobs))]
    for t in threads:
        t.start()
    start.wait()
    t0 = time.perf_counter()
    for t in threads:
        t.join()
    return out, time.perf_counter() - t0


def test_lone_states_of_several_contexts_run_side_by_side(gpu_context):
    """Four contexts with a D = 32 state each (28 CTAs): the device holds all four at once, so four
    threads take far less than four times the time of one; and no call's trajectory time holds another's."""
    from rcmps_b200 import _lib
    state = _state(32, False, 3)
    contexts = [_lib.Context(0) for _ in range(4)]

    def job(ctx):
        return lambda: [(_quartic(ctx, [state], window=30.0)[0][:3], ctx.timings()[0]) for _ in range(6)]
    for ctx in contexts:
        job(ctx)()
    alone, t1 = _in_threads([job(contexts[0])])
    together, t4 = _in_threads([job(ctx) for ctx in contexts])
    want = alone[0][0][0]
    for calls in together:
        for got, _ in calls:
            assert got[0] == want[0] and np.array_equal(got[1], want[1]) and np.array_equal(got[2], want[2])
    assert t4 < 2.5 * t1
    assert np.median([ms for calls in together for _, ms in calls]) < 2.0 * np.median([ms for _, ms in alone[0]])


def test_contexts_with_states_of_several_sizes(gpu_context):
    """Lone states, a few states per launch and one team per state from six contexts at once: the
    bits of each alone."""
    from rcmps_b200 import _lib
    work = [[_state(d, i % 2 == 1, 90 + i) for i in range(n)] for d, n in
            ((16, 1), (16, 40), (64, 1), (64, 3), (96, 1), (32, 2))]
    contexts = [_lib.Context(0) for _ in work]
    want = [_quartic(ctx, states) for ctx, states in zip(contexts, work)]
    jobs = [lambda ctx=ctx, states=states: [_quartic(ctx, states) for _ in range(5)]
            for ctx, states in zip(contexts, work)]
    for calls, ref in zip(_in_threads(jobs)[0], want):
        for got in calls:
            for g, w in zip(got, ref):
                assert g[0] == w[0] and np.array_equal(g[1], w[1]) and np.array_equal(g[2], w[2])


@pytest.mark.parametrize("d", [20, 50])
def test_ode_channel_groups(gpu_context, d):
    """The 26-channel system over 8 (dp 32) and 4 (dp 64) channel groups against the oracle."""
    from rcmps_b200 import objective
    r, k, rho = _state(d, False, 70 + d)
    q = O.left_canonical_q(r, k)
    got = objective.evaluate_phi4(r, q, rho, 1.5, half_window=0.5, n_quad=8)
    ref = O.evaluate_phi4(r, q, rho, 1.5, half_window=0.5, n_quad=8)
    assert (got["stats"]["accepted"], got["stats"]["rejected"]) == (ref["stats"]["accepted"], ref["stats"]["rejected"])
    assert abs(got["value"] - ref["value"]) <= 1e-10 * max(1.0, abs(ref["value"]))
    for name in ("covector", "environment"):
        assert np.linalg.norm(got[name] - ref[name]) <= 1e-10 * max(1.0, np.linalg.norm(ref[name]))
