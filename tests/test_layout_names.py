"""Optimizer.layout() names the epoch kernel of every flag set the library returns."""
import pytest

import test_abi


@pytest.mark.parametrize("flags,dims,expect", [
    (1 | 256 | 32, 2, {"lane_major": True, "kernel": "sgd_epoch_pool<2, false>", "eight_negatives": False}),
    (1 | 256 | 8, 4, {"generic_rule": True, "kernel": "sgd_epoch_pool<4, true>"}),
    (1 | 512, 6, {"kernel": "sgd_epoch_rows<6>"}),
    (1024 | 16 | 4 | 64, 1, {"lane_major": False, "renamed": True, "twelve_negatives": True,
                             "task_order": "row blocks", "kernel": "sgd_epoch_dram<1>"}),
    (2, 1, {"lane_major": False, "kernel": "sgd_epoch_kernel2<1, false, 8, 4, false>"}),
    (8, 3, {"kernel": "sgd_epoch_kernel2<3, true, 4, 5, false>"}),
    (8, 5, {"kernel": "sgd_epoch_anydim<true>"}),
])
def test_kernel_names(ub, monkeypatch, flags, dims, expect):
    test_abi.test_layout_flags_decoded_without_gpu(ub, monkeypatch, flags, dims, expect)
