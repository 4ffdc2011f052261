"""Matrix memory of one position: value dimensions at the edges of how a CTA's state rows are dealt to its warps (24 rows, three per warp, and
25; 72, nine per warp, and 73, which take a second trip), against the plain implementation."""
import numpy as np
import pytest

import ctox_llm_b200 as ctox
import vasanex_oracle
import vasanex_util as vasanex

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("vdim", [64, 191, 192, 575, 576])
def test_single_tokens(tmp_path, vdim):
    config, tensors = vasanex.model([vasanex.mlstm(heads=2, dim=36, vdim=vdim), vasanex.mlstm(heads=1, dim=300, vdim=vdim)], seed=vdim)
    tokens = [int(t) for t in np.random.default_rng(0).integers(0, config["vocab"], 12)]
    want, _ = vasanex_oracle.forward(config, tensors, tokens)
    be = ctox.B200Backend(0)
    ex = ctox.open_model(vasanex.write_model(str(tmp_path / "m"), config, tensors), backend=be, dtype="float32", max_context_tokens=64)
    try:
        got = np.concatenate([ex.extend([t], [0]) for t in tokens])
    finally:
        ex.unload()
        be.close()
    e = vasanex.row_errors(got, want)  # 32-bit sums in another order, as in the tests of the models
    assert e.max() < 3e-5 and e.mean() < 1e-5
