"""Calls of different sizes from several threads at once: kernels whose shared memory grows with the
number of groups (group means, the histogram kernel's plans, the CSR transpose) are set up by one
thread while another launches them. Every call succeeds with the result it gives alone."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _together(jobs):
    """Runs the jobs in a thread each; what they raised."""
    errors, start = [], threading.Barrier(len(jobs))

    def body(job):
        start.wait()
        try:
            job()
        except Exception as e:  # reported by the caller's thread
            errors.append(repr(e))

    threads = [threading.Thread(target=body, args=(j,)) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    return errors


def _counts(n_rows, n_cols):
    from hpdex_gb300.resident import ResidentMatrix
    rng = np.random.default_rng(1)
    data = rng.integers(1, 30, n_rows * n_cols).astype(np.float32)
    return ResidentMatrix(data, np.tile(np.arange(n_rows, dtype=np.int64), n_cols),
                          np.arange(n_cols + 1, dtype=np.int64) * n_rows, n_rows)


def _groups(n_rows, n_groups):
    return np.random.default_rng(n_groups).permutation(np.arange(n_rows) % n_groups).astype(np.int32)


def test_group_means_of_different_group_counts():
    m = _counts(12_000, 40)
    jobs = []
    for G in (50, 5_000, 8_000):
        gid = _groups(12_000, G)
        alone = m.group_mean(gid, G)

        def job(gid=gid, G=G, alone=alone):
            for _ in range(300):
                np.testing.assert_array_equal(m.group_mean(gid, G), alone)
        jobs.append(job)
    assert not _together(jobs)


def test_integer_plans_of_different_group_counts():
    """Histogram-kernel launches of 54, 73 and 110 KB (each recorded anew after a switch)."""
    m = _counts(2_000, 3_600)
    jobs = []
    for T in (20, 220, 332):
        plan = m.plan(_groups(2_000, T + 1), T, zero_handling="min")
        plan.run()
        assert plan.timings()[1] == 3  # group ids, histogram kernel, rank kernel
        alone = [x.copy() for x in plan.download()]

        def job(plan=plan, alone=alone):
            for k in range(200):
                plan.set_histogram(False)
                plan.set_histogram(True)
                plan.run()
                if k % 50 == 0:
                    for a, b in zip(plan.download(), alone):
                        np.testing.assert_array_equal(a, b)
        jobs.append(job)
    assert not _together(jobs)


def test_csr_transposes_of_different_widths():
    from hpdex_gb300.resident import ResidentMatrix
    jobs = []
    for cols in (200, 15_000, 38_000):  # counters of 800 bytes, 60 and 152 KB
        rng = np.random.default_rng(cols)
        rows, per = 300, 40
        genes = np.concatenate([np.sort(rng.choice(cols, per, replace=False)) for _ in range(rows)]).astype(np.int64)
        data = rng.integers(1, 9, genes.size).astype(np.float32)
        want = np.bincount(genes, weights=data, minlength=cols) / rows

        def job(cols=cols, genes=genes, data=data, want=want):
            for _ in range(60):
                m = ResidentMatrix.from_csr(data, genes, np.arange(rows + 1) * per, rows, cols)
                np.testing.assert_array_equal(m.group_mean(np.zeros(rows, np.int32), 1), want)
                m.close()
        jobs.append(job)
    assert not _together(jobs)
