"""The batched solver's launch shape for few small problems: around 1024 rows,
from where a cluster of blocks has fewer rows a thread than one block.  Checked
as every launch shape is: assembled values bit-exact, solutions to 1e-9,
iterations +-2."""
import numpy as np
import pytest

from test_gpu_batch import check_against_oracle, small_batch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits", [64, 32])
@pytest.mark.parametrize("sizes", [[15], [32], [33], [34], [33, 15, 33, 8], [34, 15, 33, 8]], ids=str)
def test_few_small_problems(cuda, sizes, bits):
    B, ref, _ = small_batch(sizes, bc=True)
    B.set_precision(bits)
    B.solve(100000, 1e-10)
    if bits == 64:
        check_against_oracle(B, ref)
    else:
        u, it, res = B.results()
        assert (res <= 1e-10).all() and (it >= 0).all()
        want = np.concatenate([r["u"] for r in ref])
        assert np.linalg.norm(u - want) <= 1e-8 * np.linalg.norm(want)
