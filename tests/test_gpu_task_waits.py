"""The bounded waits of the tile-task inverse when its schedule cannot finish: every CTA that waits
leaves, the call returns a status and the device stays usable."""
import numpy as np
import pytest

from uncertaintyte_b200 import native

pytestmark = pytest.mark.gpu


def _spd(n, seed):
    rng = np.random.default_rng(seed)
    Q = rng.standard_normal((n, n))
    return Q @ Q.T + n * np.eye(n)


def _bounded(A, poll_limit, skip_task):
    import torch
    n = A.shape[0]
    lda = (n + 7) & ~7
    buf = torch.zeros((n, lda), dtype=torch.float64, device="cuda")
    buf[:, :n] = torch.from_numpy(A)
    native.spd_inverse_tasks_bounded(buf.data_ptr(), n, lda, poll_limit, skip_task)
    torch.cuda.synchronize()
    return buf[:, :n].cpu().numpy().T


@pytest.mark.parametrize("kind", [1, 2, 3, 4])
def test_waiting_ctas_leave_together_on_abort(kind):
    """One task of a kind (TRSM, UPDATE, TACC, TFIN) left out: the CTAs behind it run out of polls at
    different times, so the abort flag rises while the warps of others are between two reads of it."""
    n = 1280  # 20 x 20 tiles
    tasks = native.spd_task_list(n)
    of_kind = np.flatnonzero(tasks[:, 0] == kind)
    A = _spd(n, 3)
    for at, polls in ((0, 200), (len(of_kind) // 2, 500), (len(of_kind) // 3, 2000)):
        with pytest.raises(native.UncError) as e:
            _bounded(A, polls, int(of_kind[at]))
        assert e.value.status == -4 and "ran out" in str(e.value)
    got, ref = _bounded(A, 1 << 22, -1), np.linalg.inv(A)
    assert np.max(np.abs(got - ref)) / np.max(np.abs(ref)) < 1e-11


def _resident(A, ctas):
    import torch
    n = A.shape[0]
    lda = (n + 7) & ~7
    buf = torch.zeros((n, lda), dtype=torch.float64, device="cuda")
    buf[:, :n] = torch.from_numpy(A)
    native.spd_inverse_tasks_resident(buf.data_ptr(), n, lda, ctas)
    torch.cuda.synchronize()
    return buf[:, :n].cpu().numpy()


@pytest.mark.parametrize("n", [1, 64, 65, 129, 200, 640, 1351, 2400])
def test_any_number_of_resident_ctas_completes(n):
    """One CTA (which runs the diagonal tasks and, while these wait, all others), two and three, and
    as many as fit: the same bytes."""
    A = _spd(n, n)
    full = _resident(A, 1 << 20)
    ref = np.linalg.inv(A)
    assert np.max(np.abs(full - ref)) / np.max(np.abs(ref)) < 1e-11
    for ctas in (1, 2, 3):
        np.testing.assert_array_equal(_resident(A, ctas), full)


def test_resident_arguments():
    import torch
    buf = torch.eye(8, dtype=torch.float64, device="cuda")
    for n, ctas in ((8, 0), (3585, 1), (0, 1)):
        with pytest.raises(native.UncError) as e:
            native.spd_inverse_tasks_resident(buf.data_ptr(), n, 8, ctas)
        assert e.value.status == -1
