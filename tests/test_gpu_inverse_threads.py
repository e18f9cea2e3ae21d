"""Inverse selection lists from several threads whose numbers of blocks need different amounts of shared memory, all beyond what a kernel has
without asking."""
import threading

import pytest
import torch

pytestmark = pytest.mark.gpu


def test_threads_with_different_numbers_of_blocks(native):
    g = torch.Generator("cuda").manual_seed(0)
    sizes = (4097, 12288, 6000, 9001)
    idx = {n: torch.randint(-1, n, (1, 1, 40, 8), device="cuda", generator=g).int() for n in sizes}
    want = {n: native._inverse_blocks_torch(idx[n], n, 4, 2)[:3] for n in sizes}
    torch.cuda.synchronize()
    failed = []

    def work(n):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(300):
                    got = native.inverse_blocks(idx[n], n, 4, 2)[:3]
                torch.cuda.current_stream().synchronize()
            listed = int(want[n][1][-1])
            if not (torch.equal(got[0][:listed], want[n][0][:listed]) and all(torch.equal(a, b) for a, b in zip(got[1:], want[n][1:]))):
                failed.append(n)
        except RuntimeError as e:
            failed.append(e)

    threads = [threading.Thread(target=work, args=(n,)) for n in sizes]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed
