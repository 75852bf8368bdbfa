"""Names that C callers of include/lpg.h may use stay in it."""

import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent


def test_a_caller_with_the_static_scratch_size_still_builds(tmp_path):
    src = tmp_path / "caller.c"
    src.write_text('#include "lpg.h"\n'
                   "static int words[LPG_COUNT_SEIRP_MAX_NODES * (4 + 2 * LPG_MAX_STRAINS) + 1 <="
                   " LPG_COUNT_SEIRP_STATIC_WORDS ? 1 : -1];\n"
                   "int main(void) { return words[0]; }\n")
    subprocess.run(["gcc", "-Wall", "-Werror", f"-I{ROOT / 'include'}", str(src), "-o", str(tmp_path / "caller")],
                   check=True)
