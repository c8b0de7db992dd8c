"""Kernels with a shared-memory limit above the default, launched from several
host threads with different sizes at a time."""

import threading
from fractions import Fraction

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _on_threads(jobs):
    """Run the jobs at the same time, each on a stream of its own; the failures."""
    import torch

    failed = []
    start = threading.Barrier(len(jobs))

    def work(job):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                start.wait()
                job()
                torch.cuda.current_stream().synchronize()
        except Exception as e:  # reported by the main thread
            failed.append(e)

    torch.cuda.synchronize()
    threads = [threading.Thread(target=work, args=(j,)) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    return failed


@pytest.mark.parametrize("blocks", [(12, 4), (20, 4), (20, 2)], ids=str)
def test_batches_of_different_widths(blocks):
    """12 and 20 instances of 4 columns take 52 and 87 KB in the update, 57 and
    60 KB in the reduction; against each other and against a narrow batch."""
    import realspace_exatdiagonalization_py_b200 as ed
    from realspace_exatdiagonalization_py_b200 import models
    from realspace_exatdiagonalization_py_b200.lanczos import LanczosBatch

    m = models.build_heisenberg_second_quantized_model(20, 1.0)
    data = ed.build_ed_data(m, filling_fraction=Fraction(1, 2), symmetry_group=ed.build_translation_group(m.lattice))
    dm, sset = data._device()
    dm.build_projection(sset.sqrt_stab, precisions=(64,))
    n, b = blocks
    batches = [LanczosBatch(dm, sset, [s % 20 for s in range(k)], 1, ed.LanczosParams(block=w))
               for k, w in ((n, b), (16, 4))]

    def steps(x):
        def job():
            for _ in range(40):
                x.load_start(None)  # the steps overwrite W
                x.start()
                x.iterate_span(14, False)
        return job

    alone = []
    for x in batches:
        steps(x)()
        alone.append(x.P.cpu().numpy())
    assert not _on_threads([steps(x) for x in batches])
    for x, want in zip(batches, alone):
        np.testing.assert_array_equal(x.P.cpu().numpy(), want)
