"""Rules of the CUDA sources that neither the compiler nor a run on well-behaved inputs checks."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "my_nn_engine_b200", "csrc")


def sources():
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        with open(path) as f:
            yield os.path.basename(path), re.sub(r"//[^\n]*", "", f.read())


def test_aligned_instructions_are_reached_by_whole_warps():
    """barrier.cluster.*.aligned and the loads, stores and waits of tensor memory are undefined unless the whole warp executes them together: a warp barrier
    stands right in front of each."""
    found = 0
    for name, text in sources():
        for m in re.finditer(r'asm volatile\(\s*"(?:barrier\.cluster|tcgen05\.(?:ld|st|wait))[a-z.:]*aligned', text):
            found += 1
            assert text[:m.start()].rstrip().endswith("__syncwarp();"), (name, m.group(0))
    assert found >= 8


def test_local_arrays_are_aligned_for_the_pieces_they_are_accessed_in():
    """A local array of small elements that is read or written through a wider type says so by its alignment: in registers it makes no difference, in a
    debug build or after a spill it is a misaligned access."""
    element = r"(?:T|O|OutT|ActT|__half|__nv_bfloat16|u?int8_t)"
    for name, text in sources():
        for m in re.finditer(r"reinterpret_cast<(?:const )?(?:u?int[248]|float[24]|u?int(?:32|64)_t) \*>\((\w+)", text):
            declared = list(re.finditer(r"^.*?\b%s(\[|\b)[^;\n]*" % m.group(1), text[:m.start()], re.M))
            arrays = [d.group(0).strip() for d in declared if re.match(r"\s*(?:__align__\(\d+\) )?%s (?:\w+\[\w+\], )*%s\[" % (element, m.group(1)), d.group(0))]
            assert not arrays or arrays[-1].startswith("__align__"), (name, arrays[-1])
