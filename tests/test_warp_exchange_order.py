"""The warp-cooperative reconstruction hands face records from one lane to
others through shared memory.  Votes and shuffles order no memory, so every
such hand-over needs a __syncwarp (or a block barrier) between the stores and
the loads; a missing one is a race that no run is bound to show, hence this
check of the source."""
import os
import re

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                   "quasar_b200", "csrc", "mhd_kernels.cu")


def body(text, name):
    at = re.search(r"\b%s\(const Grid& g" % name, text).start()
    start = text.index("{", at)
    depth = 0
    for k in range(start, len(text)):
        depth += {"{": 1, "}": -1}.get(text[k], 0)
        if depth == 0:
            return re.sub(r"//[^\n]*", "", text[start:k + 1])
    raise AssertionError(name)


def test_face_records_are_ordered_before_other_lanes_read_them():
    with open(SRC) as f:
        b = body(f.read(), "mp_faces_warp")
    segments = re.split(r"__syncwarp\([^)]*\)", b)
    own = [bool(re.search(r"=\s*rec \+ lane\b", s)) for s in segments]
    other = [bool(re.search(r"=\s*rec \+ f\b|\brec\[[^]]*\+ f\]", s)) for s in segments]
    assert sum(own) == 2  # phase 1 stores, phase 3 loads
    assert sum(other) >= 3  # eigen scalars, reference state, face values
    assert not any(a and c for a, c in zip(own, other))
