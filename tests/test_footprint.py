"""CPU tests of the scratch that a CreateDAG call lays out (dagc_create_footprint)."""
import pytest

import dag_compression_fast_gb300 as D


@pytest.mark.parametrize("depth,lg,gigabytes", [(13, 30, 187.8), (15, 29, 141.6), (17, 29, 185.6), (21, 28, 140.5),
                                                (21, 29, 273.7)])
def test_the_largest_inputs_fit_the_device(depth, lg, gigabytes):
    """The hash-set form's scratch when every level was deduplicated before the next was extracted: inputs that
    filled the device's 298 GB then still fit."""
    assert D.create_footprint(1 << lg, depth) <= gigabytes * 1e9


@pytest.mark.parametrize("depth,n,megabytes", [(10, 2000, 86.8), (5, 3000, 86.4), (9, 2000, 86.7)])
def test_the_brick_table_is_not_part_of_a_small_calls_need(depth, n, megabytes):
    """134 MB at depth 10, which a call takes only where there is room."""
    assert D.create_footprint(n, depth) <= megabytes * 1e6
