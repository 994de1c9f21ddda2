"""Options that a C caller gets from sgw_engine_opts_default, as every binding does."""
import inspect


def test_batches_choose_their_own_share_by_default(native):
    """The engine's chunk-list setting must not reach a batch, where the same
    field is the fewest edges of a warp's share: 0 leaves it to either."""
    assert native.default_opts().chunk_edges == 0


def test_batch_tuning_tries_the_default():
    from subway_gb300 import autotune
    assert 0 in inspect.signature(autotune.tune_batch).parameters["candidates"].default
