"""Where the adjoint's PCG keeps its vectors: the plan of d2ic_pcg_solve over meshes and column counts (CPU)."""
from __future__ import annotations

import ctypes

import pytest


@pytest.fixture
def plan(built_library):
    def of(nodes, columns, sms=152):
        blocks = ctypes.c_int(-1)
        return built_library.d2ic_pcg_plan(nodes, columns, sms, ctypes.addressof(blocks)), blocks.value
    return of


@pytest.mark.parametrize("nodes,columns,launches", [
    (7_569, 64, 1), (7_569, 512, 8), (65_536, 64, 8), (131_044, 128, 32), (263_169, 64, 32), (580_644, 32, 32),
])
def test_few_launches_stay_on_the_chip(plan, nodes, columns, launches):
    cols, blocks = plan(nodes, columns)
    assert cols >= 1 and -(-columns // cols) == launches and 1 <= blocks <= 152


@pytest.mark.parametrize("nodes,columns", [(131_044, 129), (263_169, 65), (330_625, 33), (330_625, 64), (580_644, 64)])
def test_many_launches_go_to_memory(plan, nodes, columns):
    """Large meshes with many columns: one pass over the operator for all columns is faster than more than 32
    launches that each read it."""
    assert plan(nodes, columns)[0] == 0


@pytest.mark.parametrize("nodes,sms,cols", [(589_000, 152, 1), (589_001, 152, 0), (644_809, 152, 0), (3_875, 1, 1), (3_876, 1, 0)])
def test_a_column_of_the_largest_mesh(plan, nodes, sms, cols):
    """3,875 pairs of 56 bytes in the shared memory of an SM."""
    assert plan(nodes, 1, sms)[0] == cols


@pytest.mark.parametrize("nodes,columns,blocks", [(16, 64, 1), (1_024, 1, 1), (1_025, 1, 3), (171, 6, 3), (1_681, 6, 20)])
def test_one_block_up_to_two_pairs_per_thread(plan, nodes, columns, blocks):
    assert plan(nodes, columns) == (columns, blocks)


def test_arguments_without_a_plan(plan):
    assert plan(100, 1, 0) == (0, 0) and plan(0, 1) == (0, 0) and plan(1, 0) == (0, 0)
