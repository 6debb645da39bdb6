"""Short 1D levels of different lengths running on several host threads: the
shared memory a kernel may ask for is a limit of the kernel, so one level's
launch must not lower it under another's."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_lengths_at_once():
    import bamrex_b200 as bx
    from bamrex_b200 import problems
    levels = []
    for n in (1000, 1010, 1020, 1900) * 2:  # 47 KB and 90 KB
        lev = bx.Level(1, (0, 0, 0), (n - 1, 0, 0), [0.0], [1.0], [((0, 0, 0), (n - 1, 0, 0))], bx.Parm(1, limiter=1),
                       bc_lo=[1] * 3, bc_hi=[1] * 3)
        lev.set_state(problems.random_states(1, (1, 1, n), seed=n))
        levels.append(lev)
    start, errors = threading.Barrier(len(levels)), []

    def work(lev):
        try:
            start.wait()
            for _ in range(3000):
                lev.run_async(1)
                lev.run_wait()
        except Exception as e:
            errors.append(str(e))

    threads = [threading.Thread(target=work, args=(lev,)) for lev in levels]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for lev in levels:
        assert np.isfinite(lev.get_state()).all()
        lev.close()
