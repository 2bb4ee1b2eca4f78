"""A source is recompiled when a generated class header that it includes
changes: the one-launch kernels over the direct classes include many."""
import os
import re

from hfcode_b200 import build


def test_objects_depend_on_the_class_headers_they_include():
    import sys
    sys.path.insert(0, build.CSRC)
    try:
        import gen_eri
    finally:
        sys.path.pop(0)
    out = os.path.join(build.CSRC, "generated")
    srcs = gen_eri.main(out)
    several = 0
    for s in srcs:
        want = {os.path.join(out, n) for n in re.findall(r'#include "(cls_\w+\.cuh)"', open(s).read())}
        assert want and want <= set(build._includes(s)), s
        several += len(want) > 1
    assert several == 2  # direct_all32.cu, direct_all64.cu
