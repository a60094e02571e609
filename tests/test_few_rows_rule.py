"""Which kernels for few rows are taken: the sizes at which they were measured to be slower go to the general kernel, as they did before there was
another."""

from __future__ import annotations

import pytest

from research_2_b200.csrc.build import BuildError, kernel_library


def takes(m, n, k, norm=0):
    try:
        return bool(kernel_library("few_rows").r2_few_rows_takes(m, n, k, norm))
    except BuildError as err:
        pytest.skip(str(err))


# rows, features, K, norm (0 none, 1 RMS norm, 2 LayerNorm): 1 us and more beside it
@pytest.mark.parametrize("m,n,k,norm", [
    (64, 12288, 64, 0), (33, 6144, 192, 0), (48, 10240, 128, 0), (64, 2560, 64, 0), (64, 1280, 3072, 0), (64, 256, 8192, 0),
    (17, 10240, 256, 0), (32, 8192, 512, 0), (24, 5120, 64, 0), (24, 2560, 2048, 0), (32, 1600, 4096, 0), (32, 1280, 4096, 0),
    (9, 10240, 384, 0), (16, 10240, 768, 0), (16, 2560, 2560, 0), (12, 3584, 2048, 0),
    (1, 3584, 2048, 0), (8, 2560, 4096, 0), (4, 1280, 8192, 0),
    (1, 10240, 1024, 2), (16, 12288, 64, 2), (16, 10240, 128, 1),
])
def test_sizes_that_the_other_kernel_does_faster(m, n, k, norm):
    assert not takes(m, n, k, norm)


# what a step's products are (layers of 768, 1,024 and 1,600, joint matrices of up to 9,216 features)
@pytest.mark.parametrize("m,n,k,norm", [
    (1, 2304, 768, 2), (16, 3072, 768, 2), (8, 9216, 768, 1), (8, 9216, 768, 2), (16, 4096, 1024, 2), (64, 768, 768, 0), (48, 3072, 768, 0), (64, 768, 3072, 0), (32, 1024, 4096, 0),
    (1, 6400, 1600, 0), (8, 1600, 6400, 0), (16, 4800, 1600, 0), (32, 768, 3072, 0), (64, 1024, 1024, 0), (1, 12288, 768, 0), (64, 3072, 768, 0),
])
def test_sizes_that_it_takes(m, n, k, norm):
    assert takes(m, n, k, norm)


@pytest.mark.parametrize("rows,heads,groups,by_group", [(6, 12, 6, True), (1, 12, 2, True), (148, 16, 4, True), (149, 16, 4, False), (6, 12, 1, False), (1, 32, 1, False), (6, 34, 2, False)])
def test_what_the_delta_rule_walks_over_by_row_and_group(rows, heads, groups, by_group):
    try:
        assert bool(kernel_library("state_scan").r2_delta_prepare_by_group(rows, heads, groups, 148)) is by_group
    except BuildError as err:
        pytest.skip(str(err))
