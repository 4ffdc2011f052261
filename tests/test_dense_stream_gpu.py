"""Products of one position with large dense matrices (k_dense_stream): matrices at or above its size limit, through models
whose tokens are taken one by one, against the plain implementations."""
import numpy as np
import pytest

import ctox_llm_b200 as ctox
import lomelorn_oracle
import lomelorn_util as lomelorn
import vasanex_oracle
import vasanex_util as vasanex

pytestmark = pytest.mark.gpu

# Each has at least one product of 4 MB or more with, in turn: a last vector of columns that is partly padding and a ragged second
# warp (131 and 263 vectors), the rotated output and the cache append; a row of nine vectors, 30011 rows; biases, gated pairs, two
# warps of 129 and 128 vectors; sixteen warps per row, fewer pairs of rows than CTAs; one column more than the kernel takes.
MODELS = {
    "ragged": lambda: (lomelorn_oracle, lomelorn.model([lomelorn.layer(heads=24, dim=120, rot_dim=56, vdim=40, q_rank=516, kv_rank=72,
                                                                       window=9, ff=2100)], vocab=2503, width=1046, seed=1)),
    "narrow": lambda: (lomelorn_oracle, lomelorn.model([lomelorn.layer()], vocab=30011, width=71, seed=2)),
    "gated": lambda: (vasanex_oracle, vasanex.model([vasanex.attention(heads=16, kv_heads=2, dim=80, vdim=72, window=7, ff=1101),
                                                     vasanex.mlstm(heads=2, dim=300, vdim=516, ff=1024)], vocab=1100, width=2056, seed=3)),
    "long_rows": lambda: (lomelorn_oracle, lomelorn.model([lomelorn.layer(ff=20480), lomelorn.layer(ff=20481)], width=250, seed=4)),
}


@pytest.fixture(scope="module")
def be():
    b = ctox.B200Backend(0)
    yield b
    assert b.allocated_bytes() == 0
    b.close()


@pytest.mark.parametrize("name", sorted(MODELS))
def test_single_tokens(be, tmp_path, name):
    oracle, (config, tensors) = MODELS[name]()
    tokens = [int(t) for t in np.random.default_rng(0).integers(0, config["vocab"], 12)]
    want, _ = oracle.forward(config, tensors, tokens)
    ex = ctox.open_model(lomelorn.write_model(str(tmp_path / "m"), config, tensors), backend=be, dtype="float32", max_context_tokens=64)
    try:
        got = np.concatenate([ex.extend([t], [0]) for t in tokens])
        again = []
        ex.reset_session()
        for t in tokens:
            again.append(ex.extend([t], [0]))
    finally:
        ex.unload()
    # sums of at most 20481 products in 32 bits through at most six products in a row: 3e-5 as in the tests of the models
    e = lomelorn.row_errors(got, want)
    assert e.max() < 3e-5 and e.mean() < 1e-5
    np.testing.assert_array_equal(got, np.concatenate(again))
