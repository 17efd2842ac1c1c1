"""The host's knowledge of a sparse schedule (torch_binding.cpp, which leaves the merge kernel out by it) against the integer
statement of the schedule: whether requests of one length are split, for every batch and number of partitions of the range."""
import pytest

from oracle import scheduler


@pytest.mark.parametrize("topk", [64, 128, 512, 2048, 2112, 4096])
def test_host_rule_agrees_with_the_schedule(topk):
    from flashmla_windows_linux_sm120_b200._cabi import native
    seen = set()
    for parts in (1, 2, 3, 9, 18, 24, 37, 49, 74, 148):
        for b in [*range(1, 40), 60, 63, 64, 65, 73, 74, 75, 127, 128, 147, 148, 149, 222, 296, 500]:
            _, ns = scheduler.schedule_cut_ref([0] * b, parts, topk)
            whole = ns[-1] == b
            assert native.splits_nothing(b, topk, parts) == whole, (b, parts)
            seen.add(whole)
    assert seen == ({True} if topk == 64 else {True, False})           # one block cannot be split
