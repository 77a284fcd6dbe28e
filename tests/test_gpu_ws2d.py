"""k_integrate2d_ws and, under the delj trick, k_integrate2d_delj (each sweep's
factors or coefficients on other warps than its solves) against
k_integrate2d, which runs them one after the other: the same bits, at the
edges of their warps of lines, load batches and ring of step scalars, and in
both forms of the solve."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _sets(n, steps, seed):
    """IM sets of about `steps` steps with growth, migration and a set without
    migration (exact zero couplings at the boundary rows)."""
    rng = np.random.default_rng(seed)
    p = np.stack([rng.uniform(0.3, 0.7, n), rng.uniform(0.3, 3, n), rng.uniform(0.3, 3, n),
                  np.full(n, steps * 1e-4), rng.uniform(9, 10, n), rng.uniform(0, 9, n)], axis=1)
    p[-1, 4:] = 0
    return p


def _both(L, rec):
    from dadi_gb300 import batch
    eng = batch.Batch2D((L,), (4, 4))
    out = []
    for threads in (0, 128):  # 128: one warp for both
        eng.threads = threads
        phis, status = eng.integrate(rec)
        assert int(status.abs().sum()) == 0
        out.append(phis[0].cpu().numpy())
    return out


@pytest.mark.parametrize("L", [3, 4, 5, 12, 13, 31, 32, 33, 63, 64, 65, 96, 97, 128, 129, 159,
                               160, 161])
def test_same_bits_at_every_warp_count(cuda_lib, L):
    from dadi_gb300 import batch
    got, want = _both(L, batch.im_instances(_sets(3, 40 if L < 100 else 18, L)))
    assert np.array_equal(got, want)


@pytest.mark.parametrize("L", [3, 4, 6, 7, 31, 33, 64, 65, 97, 129, 157, 160])
def test_same_bits_under_the_delj_trick(cuda_lib, monkeypatch, L):
    from dadi_gb300 import _lib, batch, integration
    monkeypatch.setattr(integration, "use_delj_trick", True)
    rec = batch.im_instances(_sets(3, 36 if L < 40 else 6, L))
    rec["gamma"][0, 0, 1] = 8.0
    if L == 160:  # beyond the delj trick's shared memory with one warp for both: refused
        with pytest.raises(_lib.DgbError):
            _both(L, rec)
        return
    got, want = _both(L, rec)
    assert np.array_equal(got, want)


@pytest.mark.parametrize("delj", [False, True])
def test_same_bits_across_the_scalar_ring_and_masks(cuda_lib, monkeypatch, delj):
    """Schedules of 0 to 130 steps in one queue, frozen axes and suppressed
    mutations, selection."""
    from dadi_gb300 import batch, integration
    monkeypatch.setattr(integration, "use_delj_trick", delj)
    p = _sets(24, 60, 1)
    p[:, 3] *= np.linspace(0, 2.2, 24)
    p[8:16, 4:] = 0
    rec = batch.im_instances(p)
    rec["frozen"][8:16] = np.arange(8) % 4
    rec["nomut"][12:20] = np.arange(8) % 4
    rec["gamma"][::3, 0, 1] = -30.0
    got, want = _both(47, rec)
    assert np.array_equal(got, want)


def test_same_bits_where_the_solves_form_a_again(cuda_lib):
    """More CTAs than have their coefficients in L2."""
    from dadi_gb300 import batch
    got, want = _both(130, batch.im_instances(_sets(170, 6, 2)))
    assert np.array_equal(got, want)


@pytest.mark.parametrize("L", [3, 5, 31, 33, 64, 65, 97, 112, 113])
@pytest.mark.parametrize("selection", [False, True])
def test_adjoint_walk_on_groups_of_warps(cuda_lib, L, selection):
    """The trajectory-mode backward walk (k_adjoint2d_ws up to 112 points)
    against the segment-mode walk, which runs its parts one after the other:
    the same bits, with and without parameters that gamma and h depend on,
    frozen axes, schedules of none to more steps than the scalars' ring."""
    import torch
    from dadi_gb300 import batch
    eng = batch.Batch2D((L,), (4, 4))
    eng.cluster_adjoint, eng.cluster_forward = 0, False
    p = _sets(6, 44 if L < 70 else 20, L)
    p[0, 3] = 0.0
    p[2:4, 4:] = 0
    rec = batch.im_instances(p)
    rec["gamma"][:, 0, 1], rec["h"][:, 1, 1] = 2.0, 0.3
    rec["frozen"][2:4] = [1, 2]
    rec["nomut"][4] = 1
    seeds = batch.im_seeds(6)
    if selection:
        seeds["dform"][1:, 4, 0, 0] = 1.0   # gamma of population 1 moves with s
        seeds["dform"][1:, 7, 0, 5] = -0.5  # h of population 2 with m21
    data = torch.ones(5, 5, dtype=torch.float64, device="cuda")
    got = [eng.loglik_and_grad(p, data, scale=10.0, rec=rec, seeds=seeds, trajectory=t)[1].cpu().numpy()
           for t in (True, False)]
    assert np.isfinite(got[1]).all() and np.abs(got[1]).max() > 0
    assert np.array_equal(got[0], got[1])


def _form(lib, L, n, delj=False):
    """(CTAs per SM, whether a is kept) of the split kernels' launch over n
    grids of L points, or None where k_integrate2d serves."""
    import ctypes
    import torch
    from dadi_gb300 import _lib
    ctas, keep = ctypes.c_int(), ctypes.c_int()
    rc = lib.dgb_probe_split2d(L, n, int(delj), lib.dgb_workspace_bytes(1, 2, L, n),
                               ctypes.byref(ctas), ctypes.byref(keep))
    if rc != 0:
        assert rc == _lib.DGB_ERR_UNSUPPORTED
        return None
    return ctas.value / torch.cuda.get_device_properties(0).multi_processor_count, keep.value


@pytest.mark.parametrize("L,n,keep", [(31, 2400, 1), (64, 1500, 1), (80, 920, 1), (90, 920, 0),
                                      (100, 920, 0), (128, 170, 0), (130, 170, 0)])
def test_same_bits_with_full_sms(cuda_lib, L, n, keep):
    """Several CTAs per SM (as many as shared memory and registers hold), and
    both forms of the solve at three to five warps of lines."""
    from dadi_gb300 import batch
    per_sm, kept = _form(cuda_lib, L, n)
    assert kept == keep
    assert per_sm >= (3 if L <= 64 else 2 if L <= 100 else 1)
    got, want = _both(L, batch.im_instances(_sets(n, 4, 3)))
    assert np.array_equal(got, want)


@pytest.mark.parametrize("L,n", [(3, 160), (31, 153), (31, 700), (32, 400), (33, 400), (47, 310),
                                 (64, 400)])
@pytest.mark.parametrize("spread", [0.0, 1.0, 12.0])
def test_same_bits_where_ctas_choose_to_run(cuda_lib, L, n, spread):
    """A few items per SM: more CTAs are launched than SMs, and those beyond
    run if the schedules are of similar length (all alike; from none to twice
    the mean; one of 13 times the others)."""
    from dadi_gb300 import batch
    per_sm, kept = _form(cuda_lib, L, n)
    assert per_sm > 1 and kept
    p = _sets(n, 6, 4)
    if spread == 1.0:
        p[:, 3] *= np.linspace(0, 2, n)
    elif spread:
        p[n // 2, 3] *= 1 + spread
    got, want = _both(L, batch.im_instances(p))
    assert np.array_equal(got, want)


def test_checkpoints_where_ctas_choose_to_run(cuda_lib):
    """The same launch with checkpoints, from which gradients are walked back:
    the bits of the gradients from k_integrate2d's."""
    import torch
    from dadi_gb300 import batch
    p = _sets(200, 9, 5)
    p[:, 3] *= np.linspace(0.2, 2, 200)
    data = torch.ones(5, 5, dtype=torch.float64, device="cuda")
    out = []
    for threads in (0, 128):
        eng = batch.Batch2D((31,), (4, 4))
        eng.threads = threads
        ll, grad, _ = eng.loglik_and_grad(p, data, scale=10.0)
        out.append((ll.cpu().numpy(), grad.cpu().numpy()))
    assert np.isfinite(out[1][1]).all()
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])


def test_end_of_the_split_kernels_range(cuda_lib):
    """159 points are the last that the split kernels take."""
    for delj in (False, True):
        assert _form(cuda_lib, 159, 3, delj) and _form(cuda_lib, 160, 3, delj) is None


def _gradient(L, steps, selection, trajectory):
    import torch
    from dadi_gb300 import batch
    eng = batch.Batch2D((L,), (4, 4))
    eng.cluster_adjoint, eng.cluster_forward = 0, False
    p = _sets(5, steps, L)
    rec, seeds = batch.im_instances(p), batch.im_seeds(5)
    rec["frozen"][3], rec["nomut"][2] = 2, 1
    if selection:
        seeds["dform"][1:, 4, 0, 0] = 1.0
    data = torch.ones(5, 5, dtype=torch.float64, device="cuda")
    return eng.loglik_and_grad(p, data, scale=10.0, rec=rec, seeds=seeds,
                               trajectory=trajectory)[1].cpu().numpy()


@pytest.mark.parametrize("L", [103, 104, 105, 106])
def test_adjoint_walk_at_the_end_of_its_range(cuda_lib, L):
    """The last grids that k_adjoint2d_ws takes and the first that it does not
    (the workspace query tells them apart) against the segment-mode walk."""
    split = cuda_lib.dgb_adjoint2d_traj_ws_bytes(L, 2) > 256 + 2 * 8 * L * L
    assert split == (L <= 105)
    for selection in (False, True):
        got, want = [_gradient(L, 20, selection, t) for t in (True, False)]
        assert np.isfinite(want).all() and np.abs(want).max() > 0
        assert np.array_equal(got, want)
