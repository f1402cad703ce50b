"""What the kernels' sources promise and no single launch shows."""
import os
import re

import llm_infer_rust_b200.kernels.build as build


def test_launch_limits_do_not_follow_the_launches():
    """A kernel's limit of shared memory is set once, to one size.  Kept in a number that grows with the launches it could be set
    by two threads in the wrong order, the smaller size last and the larger one remembered; launches in between then fail."""
    seen = 0
    for name in sorted(os.listdir(build.CSRC)):
        if name.endswith(".cu"):
            with open(os.path.join(build.CSRC, name)) as f:
                text = f.read()
            seen += len(re.findall(r"\bstatic bool configured\b", text))
            grows = re.findall(r"\bstatic (?:size_t|int|unsigned|long long) configured\b.*", text)
            assert not grows, f"{name}: {grows}"
    assert seen > 5
