"""The autotuner's default search tries no two settings that the library runs alike."""
import importlib


def test_search_values_differ_in_effect(pkg):
    tuning = importlib.import_module("jax-cpfem_gb300.tuning")
    values = dict(tuning.SEARCH)
    assert set(values) <= set(tuning.DEFAULT)
    assert all(len(set(v)) == len(v) and tuning.DEFAULT[k] in v for k, v in values.items())
    # the dense coarse operator takes levels of at most 256 nodes, whatever larger bound is given
    assert len({min(v, 256) for v in values["local_nodes"]}) == len(values["local_nodes"])
    # 0 is one block per SM (152), which a larger count is clamped to
    assert len({min(v, 152) or 152 for v in values["grid_blocks"]}) == len(values["grid_blocks"])
