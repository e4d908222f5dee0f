"""The schedules of the attention kernels, run as a host model (one thread per role, the same
barriers, parities and issue order as ``csrc/attention_fwd2_impl.cuh``, ``csrc/attention_bwd2_impl.cuh`` and
``csrc/attention_bwd3_impl.cuh``, random delays in every role):
every sweep length must terminate and give the directly computed results."""
import numpy as np
import pytest

from distdl_b200.ops import attention_model as model

BT, D = 8, 4
SCALE = 0.5
C = SCALE * 1.4426950408889634


def _tiles(rng, n):
    return [rng.standard_normal((BT, D)) for _ in range(n)]


def _p(q, k, l2, mask):
    p = np.exp2(q @ k.T * C - l2[:, None])
    return np.where(mask, 0.0, p) if mask is not None else p


UPPER = np.arange(BT)[None, :] > np.arange(BT)[:, None]          # key later than query


@pytest.mark.parametrize("iters,diag_at", [(1, (0,)), (2, (0,)), (3, ()), (4, (0, 2)), (7, (0,)), (12, ())])
def test_dkdv_schedule_terminates_and_matches(iters, diag_at):
    rng = np.random.default_rng(iters)
    Q, dO = _tiles(rng, iters), _tiles(rng, iters)
    K, V = _tiles(rng, 2)
    l2 = [rng.standard_normal(BT) + 2 for _ in range(iters)]
    dl = [rng.standard_normal(BT) for _ in range(iters)]
    dK = np.zeros((BT, D))
    dV = np.zeros((BT, D))
    for it in range(iters):
        p = _p(Q[it], K, l2[it], UPPER if it in diag_at else None)          # [query, key]
        ds = p * (dO[it] @ V.T - dl[it][:, None]) * SCALE
        dV += p.T @ dO[it]
        dK += ds.T @ Q[it]
    for seed in range(3):
        got_dk, got_dv = model.dkdv_tile(Q, dO, K, V, l2, dl, SCALE, causal_diag_at=diag_at, seed=seed)
        assert np.allclose(got_dv, dV, rtol=1e-10, atol=1e-10), (iters, seed)
        assert np.allclose(got_dk, dK, rtol=1e-10, atol=1e-10), (iters, seed)


@pytest.mark.parametrize("nblocks,causal", [(1, True), (2, True), (3, False), (4, True), (6, False), (9, True)])
def test_dq_schedule_terminates_and_matches(nblocks, causal):
    rng = np.random.default_rng(100 + nblocks)
    (Q, dO), K, V = _tiles(rng, 2), _tiles(rng, nblocks), _tiles(rng, nblocks)
    l2, dl = rng.standard_normal(BT) + 2, rng.standard_normal(BT)
    diag = nblocks - 1 if causal else None
    dQ = np.zeros((BT, D))
    for jj in range(nblocks):
        p = _p(Q, K[jj], l2, UPPER if jj == diag else None)
        ds = p * (dO @ V[jj].T - dl[:, None]) * SCALE
        dQ += ds @ K[jj]
    for seed in range(3):
        got = model.dq_tile(Q, dO, K, V, l2, dl, SCALE, causal_diag_at=diag, seed=seed)
        assert np.allclose(got, dQ, rtol=1e-10, atol=1e-10), (nblocks, seed)


def test_a_wrong_parity_is_caught():
    """The model has teeth: waiting for the Q tile of the NEXT iteration with the parity of this one
    (the mistake the per-stage phase arithmetic guards against) ends in a bounded wait that runs out."""
    rng = np.random.default_rng(5)
    iters = 4
    Q, dO = _tiles(rng, iters), _tiles(rng, iters)
    K, V = _tiles(rng, 2)
    l2 = [np.zeros(BT) for _ in range(iters)]
    dl = [np.zeros(BT) for _ in range(iters)]
    real_wait = model.MBarrier.wait

    def wrong(self, parity):
        return real_wait(self, parity ^ 1 if self.name == "q_full[1]" else parity)
    old_limit = model.WAIT_LIMIT_S
    model.MBarrier.wait, model.WAIT_LIMIT_S = wrong, 0.5
    try:
        with pytest.raises(model.PipelineStuck):
            model.dkdv_tile(Q, dO, K, V, l2, dl, SCALE)
    finally:
        model.MBarrier.wait, model.WAIT_LIMIT_S = real_wait, old_limit


def test_a_softmax_warp_that_lags_an_iteration_behind():
    """One softmax warp far behind the others.  The dK / dV schedule cannot let any warp run a whole
    iteration ahead (dP of the next iteration waits for dS of this one).  The dQ schedule can: S and
    dP of the next key tile are issued early, so a fast warp reaches its next "dS written" arrival
    while the slow one has not arrived for this tile; with one barrier per dP buffer that arrival
    belongs to the other buffer's phase, with a single barrier it completes the wrong phase and dQ of
    this tile is formed from a dS tile with columns missing."""
    rng = np.random.default_rng(9)
    n = 5
    Q, dO = _tiles(rng, n), _tiles(rng, n)
    K, V = _tiles(rng, 2)
    l2 = [rng.standard_normal(BT) + 2 for _ in range(n)]
    dl = [rng.standard_normal(BT) for _ in range(n)]
    dK, dV = np.zeros((BT, D)), np.zeros((BT, D))
    for it in range(n):
        p = _p(Q[it], K, l2[it], None)
        dV += p.T @ dO[it]
        dK += (p * (dO[it] @ V.T - dl[it][:, None]) * SCALE).T @ Q[it]
    got_dk, got_dv = model.dkdv_tile(Q, dO, K, V, l2, dl, SCALE, slow_warp=2)
    assert np.allclose(got_dk, dK) and np.allclose(got_dv, dV)
    (q, do), Ks, Vs = _tiles(rng, 2), _tiles(rng, n), _tiles(rng, n)
    dQ = sum((_p(q, Ks[j], l2[0], None) * (do @ Vs[j].T - dl[0][:, None]) * SCALE) @ Ks[j] for j in range(n))
    assert np.allclose(model.dq_tile(q, do, Ks, Vs, l2[0], dl[0], SCALE, slow_warp=1), dQ)
    assert not np.allclose(model.dq_tile(q, do, Ks, Vs, l2[0], dl[0], SCALE, slow_warp=1, ds_full_buffers=1), dQ)


def _pair_case(qp, causal, nkv, second=True):
    rng = np.random.default_rng(50 + qp)
    n = (2 * qp + 1, 2 * qp + 2) if causal else (nkv, nkv)
    n = n if second else (n[0], 0)
    diag = (2 * qp, 2 * qp + 1) if causal else (None, None)
    Q = _tiles(rng, 2)
    K = [rng.standard_normal((BT, D)) * (1 + 4 * j) for j in range(nkv)]        # later blocks score higher
    V = _tiles(rng, nkv)
    want_o, want_l = np.zeros((2, BT, D)), np.zeros((2, BT))
    for t in range(2 if second else 1):
        s = np.concatenate([Q[t] @ K[j].T for j in range(n[t])], axis=1) * SCALE
        if causal:
            cols = np.arange(n[t] * BT)[None, :]
            s = np.where(cols > (diag[t] * BT + np.arange(BT))[:, None], -np.inf, s)
        m = s.max(axis=1, keepdims=True)
        e = np.exp(s - m)
        want_o[t] = (e / e.sum(axis=1, keepdims=True)) @ np.concatenate(V[:n[t]], axis=0)
        want_l[t] = (m + np.log(e.sum(axis=1, keepdims=True)))[:, 0]
    return (Q, K, V, n, SCALE, diag), want_o, want_l


@pytest.mark.parametrize("own_p", [False, True])
@pytest.mark.parametrize("qp,causal,nkv,second", [(0, True, 2, True), (1, True, 4, True), (3, True, 8, True), (2, True, 6, False),
                                                  (0, False, 1, True), (0, False, 5, True), (2, False, 2, False)])
def test_forward_pair_schedule_terminates_and_matches(qp, causal, nkv, second, own_p):
    """The two-tile forward kernel, with the schedules of head dim 128 and 64: both tiles alternate on the tensor pipe, the
    causal tiles see different numbers of blocks (2 qp + 1 and 2 qp + 2), a sequence may end before the second tile, scores
    that grow from block to block force the lazy rescale of the output accumulator."""
    args, want_o, want_l = _pair_case(qp, causal, nkv, second)
    for seed in range(3):
        o, lse = model.fwd_pair(*args, own_p=own_p, seed=seed, grow_threshold=2.0)
        assert np.allclose(o, want_o, rtol=1e-9, atol=1e-9), seed
        assert np.allclose(lse, want_l, rtol=1e-9, atol=1e-9)
    # one softmax warp lagging: the next S is only issued after all four warps of a tile have read their scores (at head
    # dim 128: written their probabilities), so nobody is a whole block ahead of it
    o, lse = model.fwd_pair(*args, own_p=own_p, grow_threshold=2.0, slow_warp=(1 if second else 0, 2))
    assert np.allclose(o, want_o, rtol=1e-9, atol=1e-9) and np.allclose(lse, want_l, rtol=1e-9, atol=1e-9)


def test_probabilities_written_before_they_were_read_are_caught():
    """Without the wait for the second product of the block before, a P with columns of its own is overwritten early: the
    output is wrong, or whoever waits for a phase that has gone by never sees it."""
    args, want_o, _ = _pair_case(0, False, 9)
    old_limit, model.WAIT_LIMIT_S = model.WAIT_LIMIT_S, 0.5
    try:
        wrong = 0
        for seed in range(4):
            try:
                o, _ = model.fwd_pair(*args, own_p=True, seed=seed, grow_threshold=1e9, wait_pv=False)
                wrong += not np.allclose(o, want_o)
            except model.PipelineStuck:
                wrong += 1
        assert wrong
    finally:
        model.WAIT_LIMIT_S = old_limit


def _one_pass_case(nT, heads, causal, seed):
    """Inputs of the one-pass kernel for one kv head and its gradients, computed directly."""
    rng = np.random.default_rng(200 + seed)
    D2 = 4
    Q, dO = ([[rng.standard_normal((BT, D2)) for _ in range(nT)] for _ in range(heads)] for _ in range(2))
    K, V = ([rng.standard_normal((BT, D2)) for _ in range(nT)] for _ in range(2))
    l2, dl = ([[rng.standard_normal(BT) + add for _ in range(nT)] for _ in range(heads)] for add in (2.0, 0.0))
    dQ = [[np.zeros((BT, D2)) for _ in range(nT)] for _ in range(heads)]
    dK, dV = ([np.zeros((BT, D2)) for _ in range(nT)] for _ in range(2))
    for h in range(heads):
        for i in range(nT):
            for j in range(i + 1 if causal else nT):
                p = _p(Q[h][i], K[j], l2[h][i], UPPER if causal and i == j else None)
                ds = p * (dO[h][i] @ V[j].T - dl[h][i][:, None]) * SCALE
                dQ[h][i] += ds @ K[j]
                dK[j] += ds.T @ Q[h][i]
                dV[j] += p.T @ dO[h][i]
    return (Q, dO, K, V, l2, dl, SCALE, causal), (dQ, dK, dV)


def _agree(got, want):
    return all(np.allclose(a, b, rtol=1e-9, atol=1e-9) for g, w in zip(got, want) for a, b in zip(g, w))


@pytest.mark.parametrize("roomy", [True, False])
@pytest.mark.parametrize("nT,heads,split,causal,resident", [
    (1, 1, 1, True, 1), (1, 3, 3, False, 2), (2, 1, 1, True, 2), (3, 1, 1, False, 3), (5, 1, 1, True, 2),
    (4, 2, 1, True, 4), (3, 4, 4, True, 3), (3, 4, 2, False, 6)])
def test_one_pass_schedule_terminates_and_matches(nT, heads, split, causal, resident, roomy):
    """Key tiles that start together or one after the other, heads of a group in one CTA or spread over several: every
    wait ends, and no sum of dQ, dK or dV is read before it is complete or added out of turn."""
    args, want = _one_pass_case(nT, heads, causal, nT)
    for seed in range(2):
        got = model.one_pass(*args, roomy, split=split, resident=resident, seed=seed)
        assert _agree([sum(got[0], []), *got[1:]], [sum(want[0], []), *want[1:]]), seed


def test_one_pass_without_turns_is_caught():
    """The first key tile stores where the others add: without the order of the turns the sums are wrong, or whoever
    waits for a number of parts never sees it."""
    args, want = _one_pass_case(4, 1, False, 9)
    old_limit, model.WAIT_LIMIT_S = model.WAIT_LIMIT_S, 0.5
    try:
        wrong = 0
        for seed in range(4):
            try:
                got = model.one_pass(*args, True, resident=4, seed=seed, wait_turns=False)
                wrong += not _agree([sum(got[0], []), *got[1:]], [sum(want[0], []), *want[1:]])
            except (model.PipelineStuck, RuntimeError):
                wrong += 1
        assert wrong
    finally:
        model.WAIT_LIMIT_S = old_limit
