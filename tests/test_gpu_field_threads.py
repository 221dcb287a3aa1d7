"""Fields of several solves read at once from several threads: large ones share the library's pinned pieces."""
import threading

import numpy as np
import pytest

from creep_modeling_b200 import Solve, decks

pytestmark = pytest.mark.gpu


def test_concurrent_reads_equal_single_ones(tmp_path):
    solves, want, bad = [], [], []
    for i in range(3):
        case = decks.case_c1(nsteps=1)
        case.n, case.ngrains, case.seed = 40 + 2 * i, 30, 7 + i
        s = Solve(decks.write_case(case, tmp_path / str(i)), mix=1, modal=0)
        assert s.advance(1) == 1
        solves.append(s)
        want.append({f: s.field(f) for f in ("sg", "c066mod", "wgtc")})

    def read(i):
        for _ in range(4):
            for f, ref in want[i].items():
                if not np.array_equal(solves[i].field(f), ref):
                    bad.append((i, f))

    threads = [threading.Thread(target=read, args=(i,)) for i in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for s in solves:
        s.close()
    assert not bad
