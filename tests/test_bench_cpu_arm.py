"""bench.py's CPU legs without the reference's sources: the store fields that
bench.py makes for the oracle are those of the host store builder, and the
reference arm's line says which kernels it timed."""
import sys

import numpy as np

from test_bench_reference_arm import ROOT, run_arm


def test_oracle_fields_are_the_builders():
    sys.path.insert(0, ROOT)
    import bench
    from helpers import host_store
    from sph import free_data_cpu, scenes
    for sc in [bench.workload("dam-8k", 0)[0], bench.workload("beam-4k", 0)[0]] + scenes.batch_mix(12, seed=3,
                                                                                                 n_range=(200, 2000)):
        ps, views = host_store(sc)
        made = bench.oracle_fields(sc)
        for f, want in views.items():
            if f in ("gridcell", "gridcount", "celloffset", "cellparticles"):
                continue  # made by the oracle
            assert made[f].dtype == want.dtype and made[f].tobytes() == np.ascontiguousarray(want).tobytes(), f
            assert made[f].shape == want.shape or f == "gridres", f
        free_data_cpu(ps)


def test_the_line_says_whose_kernels_it_timed():
    line = run_arm()["cpu_baseline"]
    assert ("the reference's kernels in stores" in line["sample"]) == (line["kind"] == "reference"), line
