"""Token ids and wanted places as a step takes them: looked at as a whole or one by one, accepted and refused alike."""
import numpy as np
import pytest
import torch

from transformer_b200.engine.engine import StepError, whole_numbers


def wrong(v):
    return StepError(f"{v} is wrong")


@pytest.mark.parametrize("n", [0, 1, 8, 9, 300])
def test_forms_that_are_taken(n):
    want = [(7 * i) % 50 for i in range(n)]
    forms = [want, tuple(want), np.array(want, dtype=np.int64), np.array(want, dtype=np.uint8), torch.tensor(want, dtype=torch.int32),
             [np.int32(v) for v in want], [float(v) + 0.25 for v in want], [str(v) for v in want], [torch.tensor(v) for v in want]]
    for form in forms:
        got = whole_numbers(form, 50, wrong)
        assert got.dtype == np.int64 and got.tolist() == want
    assert whole_numbers(range(n), 1000, wrong).tolist() == list(range(n))
    assert whole_numbers([True] * n, 2, wrong).tolist() == [1] * n


@pytest.mark.parametrize("n", [1, 9, 40])
@pytest.mark.parametrize("bad", [-1, 50, 1 << 40, 1 << 70, -(1 << 70)])
def test_the_first_that_does_not_fit_is_named(n, bad):
    values = [3] * n
    values[n // 2] = bad
    values[n - 1] = bad
    with pytest.raises(StepError, match=f"^{bad} is wrong$"):
        whole_numbers(values, 50, wrong)


@pytest.mark.parametrize("n", [1, 20])
def test_what_is_no_number_stays_refused(n):
    for thing, error in (("x", ValueError), (None, TypeError), ([1, 2], TypeError)):
        with pytest.raises(error):
            whole_numbers([thing] * n, 50, wrong)
