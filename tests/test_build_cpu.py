"""Every file that a source of the library includes is among the build's
dependencies, so that a change to it alone rebuilds the library."""
import os
import re

from rabbitbin_b200 import build


def test_included_files_are_dependencies():
    known = {os.path.normpath(os.path.join(build.CSRC, h)) for h in build.HEADERS}
    known.add(os.path.join(build.CSRC, "zig_tables.inc"))
    missing = set()
    for f in os.listdir(build.CSRC):
        if not f.endswith((".cu", ".cuh", ".cpp", ".h")):
            continue
        text = open(os.path.join(build.CSRC, f)).read()
        for inc in re.findall(r'^\s*#include\s+"([^"]+)"', text, re.M):
            path = os.path.normpath(os.path.join(build.CSRC, inc))
            if path not in known:
                missing.add((f, inc))
    assert not missing
