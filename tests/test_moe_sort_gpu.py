"""The sort of (row, choice) pairs by expert: every live pair once, in its expert's run of slots."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("n, E, top", [(1, 1, 1), (7, 3, 2), (257, 16, 3), (2048, 16, 4), (4096, 64, 4), (4097, 64, 4), (1365, 64, 12), (300, 65, 8), (5461, 5, 3)])
def test_every_live_pair_has_a_slot_of_its_expert(n, E, top):
    from glassbox_b200 import kernels
    gen = torch.Generator(device=DEV).manual_seed(n)
    choice = torch.randint(0, E, (n, top), dtype=torch.int32, device=DEV, generator=gen)
    positions = torch.randint(0, 9, (n,), dtype=torch.int32, device=DEV, generator=gen)
    if n > 2:
        positions[torch.randint(0, n, (n // 5 + 1,), device=DEV, generator=gen)] = -1
        choice[2, 0], choice[1, top - 1] = E, -3                       # (no experts: left out)
    if n % 2 == 0:
        choice[n // 2:] = E - 1                                        # (most pairs to one expert)
    offsets, order = torch.full((E + 1,), -1, dtype=torch.int32, device=DEV), torch.full((n * top,), -1, dtype=torch.int32, device=DEV)
    kernels._call("gb_moe_sort", choice.data_ptr(), positions.data_ptr(), n, E, top, offsets.data_ptr(), order.data_ptr(), kernels._stream())
    expert = choice.flatten().clone()
    expert[(positions < 0).repeat_interleave(top)] = -1
    live = ((expert >= 0) & (expert < E)).nonzero().flatten()
    counts = torch.bincount(expert[live].long(), minlength=E)
    assert offsets.tolist() == [0] + counts.cumsum(0).tolist()
    used = order[:len(live)]
    assert torch.equal(used.sort().values.long(), live) and (order[len(live):] == -1).all()
    assert torch.equal(expert[used.long()].long(), torch.repeat_interleave(torch.arange(E, device=DEV), counts))


@pytest.mark.parametrize("n, E, top", [(3071, 16, 1), (3072, 16, 1), (1024, 32, 3), (1535, 64, 4), (1536, 64, 4), (3073, 1, 1), (8192, 7, 2), (16385, 16, 1)])
def test_both_sides_of_the_line_sort(n, E, top):
    """Counters of all pairs below 3,072 of them (and 96 an expert) and above what a block's columns hold, columns between."""
    test_every_live_pair_has_a_slot_of_its_expert(n, E, top)


def test_threads_with_few_and_many_pairs_do_not_disturb_each_other():
    """The kernel's limit of shared memory is one for all threads of a process: a small sort beside a large one must not lower it."""
    import threading
    from glassbox_b200 import kernels
    failures = []

    def work(n, E, top):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                choice = (torch.arange(n * top, device=DEV) % E).to(torch.int32)
                positions, offsets, order = (torch.zeros(size, dtype=torch.int32, device=DEV) for size in (n, E + 1, n * top))
                for _ in range(3000):
                    kernels._call("gb_moe_sort", choice.data_ptr(), positions.data_ptr(), n, E, top, offsets.data_ptr(), order.data_ptr(),
                                  kernels._stream())
                torch.cuda.current_stream().synchronize()
                assert offsets.tolist() == [i * n * top // E for i in range(E + 1)]
        except Exception as e:      # noqa: BLE001 (reported by the thread that asserts)
            failures.append(repr(e))
    threads = [threading.Thread(target=work, args=shape) for shape in ((768, 16, 4), (4096, 64, 4), (3072, 1, 1), (4096, 64, 4))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures, failures
