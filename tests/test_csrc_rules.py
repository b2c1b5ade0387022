"""Rules of the CUDA sources that neither the compiler nor a run on well-behaved inputs checks."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "my_nn_engine_b200", "csrc")


def sources():
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        with open(path) as f:
            yield os.path.basename(path), re.sub(r"//[^\n]*", "", f.read())


def test_aligned_cluster_barriers_are_reached_by_whole_warps():
    """barrier.cluster.*.aligned is undefined unless the whole warp executes it together: a warp barrier stands right in front."""
    found = 0
    for name, text in sources():
        for m in re.finditer(r'asm volatile\(\s*"barrier\.cluster\.[a-z.]*aligned', text):
            found += 1
            assert text[:m.start()].rstrip().endswith("__syncwarp();"), name
    assert found
