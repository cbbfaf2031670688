"""Kernels that may start before the kernel in front has ended read nothing
that changes before their wait: no restrict-qualified pointer to such data, as
loads through one may be moved in front of the wait."""
import re
from pathlib import Path

CSRC = Path(__file__).parents[1] / "new_repo_b200" / "csrc"
# constant after a state's creation, or written only
FREE = {"piv", "phat"}


def test_no_restrict_on_changing_data_in_kernels_that_wait():
    seen = 0
    for path in sorted(CSRC.glob("*.cu*")):
        for part in path.read_text().split("__global__")[1:]:
            body = part.split("\n}\n")[0]
            if "dep_wait();" not in body:
                continue
            seen += 1
            names = set(re.findall(r"__restrict__\s+(\w+)", body))
            assert names <= FREE, (path.name, body.split("(")[0], names)
    assert seen >= 40
