"""The tensor-core ground truth's operands are temporary: the context holds no more
device memory after a call than before it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_ground_truth_holds_nothing():
    from anqi import pipeline
    from anqi._lib import Context

    rng = np.random.default_rng(2)
    base = rng.standard_normal((20_000, 128)).astype(np.float32)
    query = rng.standard_normal((500, 128)).astype(np.float32)
    with Context(0) as ctx:
        before = ctx.device_bytes
        rk2 = rng.uniform(100.0, 180.0, len(base)).astype(np.float32)
        pipeline.rknn_ground_truth(ctx, base, query, rk2, method="tc")
        assert ctx.device_bytes == before
