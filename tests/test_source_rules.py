"""Rules of the kernel sources that no run can show."""
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

# written before a run's first kernel, by nothing while one runs
CONSTANT = ("ipx_c.vid_of[", "ipd_vertices_count", "ipd_edges_count")


def test_read_only_loads_are_of_constant_data():
    """__ldg and ld.global.nc are for data nothing writes while the grid exists.  The superstep kernels come onto the
    SMs while the one before still writes (programmatic dependent launch), so the files that hold them read through
    that path only what is constant during a run."""
    files = [os.path.join("include", "ipregel_b200", f) for f in ("api.cuh", "engine.cuh", "host.cuh")]
    files.append(os.path.join("ipregel_b200", "csrc", "pagerank_split.cu"))
    for path in files:
        text = re.sub(r"/\*.*?\*/", "", open(os.path.join(ROOT, path)).read(), flags=re.S)
        for line in text.splitlines():
            line = line.split("//")[0]
            if "__ldg(" in line or re.search(r"ld\.global[.\w]*\.nc\b", line):
                assert any(c in line for c in CONSTANT), (path, line.strip())
