"""Stage candidates of an FP32 ensemble that is large enough for the register
march: the march is a candidate of its own, so that what autotune returns, what
info reports and what set_shape takes are the kernel that runs; a batch of at
most a wave of tiles has no such candidate.  All candidates have the same bits."""
import numpy as np
import pytest

import oracle_lib as O
from core_collapse_b200 import _lib as L
from core_collapse_b200.batch import BatchSolver, collapse_ensemble
from core_collapse_b200.mhd2d import CcError

pytestmark = pytest.mark.gpu


def _batch(n, sides, precision="fp32"):
    params, states = collapse_ensemble(n, seed=2, sides=sides, precision=precision)
    b = BatchSolver(params)
    for i, s in enumerate(states):
        b.upload(i, *s)
    return b, params, states


def test_march_is_a_candidate():
    b, params, states = _batch(12, (96, 160, 192))
    with b:
        first = b.info()
        march = first["n_shapes"] - 1
        assert first["shape"] == march and march % 2 == 0          # runs it by itself
        assert first["tile_x"] == 28 and 0 < first["tile_y"] <= 126 and first["stage_ctas"] == first["stage_tiles"] > 0
        shape, ms = b.autotune(reps=3)
        tuned = b.info()
        assert tuned["shape"] == shape and ms > 0
        b.set_shape(shape)
        assert b.info() == tuned                                    # the kernel that autotune timed
        results = {}
        for k in range(first["n_shapes"]):
            b.set_shape(k)
            info = b.info()
            assert info["shape"] == k and (info["tile_x"] == 28) == (k == march)
            for i, s in enumerate(states):
                b.upload(i, *s)
            t = b.advance(4, np.zeros(len(params)))
            results[k] = [t] + [x for i in range(len(params)) for x in O.state_list(*b.download(i))]
        b.set_shape(march)
        assert b.info() == first
        for k in (-1, march + 1):
            with pytest.raises(CcError) as e:
                b.set_shape(k)
            assert e.value.code == L.CC_ERR_ARG
    for k, r in results.items():
        assert all(np.array_equal(x, y) for x, y in zip(r, results[march])), k


@pytest.mark.parametrize("n,sides,precision", [(4, (32, 48), "fp32"), (12, (96, 160, 192), "fp64")])
def test_no_march(n, sides, precision):
    b, _, _ = _batch(n, sides, precision)
    with b:
        info = b.info()
        assert info["n_shapes"] % 2 == 0 and info["shape"] == 0 and info["tile_x"] != 28
        with pytest.raises(CcError) as e:
            b.set_shape(info["n_shapes"])
        assert e.value.code == L.CC_ERR_ARG
        assert b.autotune(reps=1)[0] == b.info()["shape"] < info["n_shapes"]
