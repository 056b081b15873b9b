"""Native Float64 lines beyond 4096 points whose smallest radix leaves a stage
more butterflies than a block has threads, each such radix (2, 3, 4, 5, 7) with
its fullest and least full round, against the oracle."""
import numpy as np
import pytest

import pencilffts_gb300 as P
from test_gpu_parity import check_plan

T = P.Transforms
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [4374, 4719, 5005, 6006, 6561, 7203, 8100, 8190])
def test_native_lines_of_many_butterflies(cuda, n):
    for tr in (T.FFT(), T.RFFT(), T.R2R(T.DHT)):
        check_plan(P.PencilFFTPlan((n, 3), (tr, T.NoTransform()), np.float64, precision="native"), seed=n)
        check_plan(P.PencilFFTPlan((3, n), (T.NoTransform(), T.FFT()), np.float64, precision="native"), seed=n + 1)
    if n % 2 == 0:
        check_plan(P.PencilFFTPlan((n // 2, 5), (T.R2R(T.REDFT01), T.NoTransform()), np.float64, precision="native"), seed=n)
