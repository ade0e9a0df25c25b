"""A chained kernel starts while the kernel before it still writes.  Its
__restrict__ parameters -- memory that nobody writes while it runs -- may only
be tables that are at least two launches old: the descriptors and the matrices
of a call (source check, no GPU)."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "nicp_b200", "csrc")
OLD_ENOUGH = {"pairs", "frames", "explicit_KRt", "explicit_T"}


def _kernels():
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        src = open(path).read()
        for m in re.finditer(r"^__global__[^{;]*?\b(k_\w+)\(([^{;]*)\)\s*\{(.*?)^\}", src, flags=re.M | re.S):
            yield m.groups()


def test_restrict_only_on_what_is_older_than_the_kernel_before():
    chained = {name: args for name, args, body in _kernels() if re.search(r"\bchain(_wait)?\(\)", body)}
    assert {"k_zbuffer", "k_corr_tile", "k_solve", "k_publish", "k_nn_query", "k_nn_far", "k_nn_pairs",
            "k_build_planes"} <= set(chained)
    for name, args in chained.items():
        assert set(re.findall(r"__restrict__\s*(\w+)", args)) <= OLD_ENOUGH, name
