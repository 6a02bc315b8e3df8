"""The pivot tiers and batches of test_gpu_pivot_tiers.py and test_gpu_batch_rows.py with
bitset rows throughout, and batches with the three-tier rule.  Exact."""
import pytest

import test_gpu_batch_rows as rows
import test_gpu_pivot_tiers as tiers
from test_gpu_pivot_tiers import graph, want  # noqa: F401 (fixtures)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [None, (2, 7, 8, 0), (64, 65536, 4, 1024)])
def test_tier_edges(eh, graph, want, shape):  # noqa: F811
    tiers.test_tier_edges(eh, graph, want, "bs", shape)


@pytest.mark.parametrize("kind", ["symmetric", "one moved", "self-loop"])
def test_lollipops(eh, oracle, graph, kind):  # noqa: F811
    tiers.test_lollipops_by_triangles_only_where_symmetric(eh, oracle, graph, "bs", kind)


@pytest.mark.parametrize("layout", ["bs", "hybrid3"])
def test_batches(eh, oracle, layout):
    tiers.test_batch_triangles_from_the_clique_masks(eh, oracle, layout)
    rows.test_batch_pivots_of_every_kind(eh, oracle, layout)
