"""What ``csrc/build.py`` compiles and where the package keeps it (no compiler and no GPU needed)."""

import fnmatch
import tomllib
from pathlib import Path

from cornstarch_b200.csrc import build as B


def test_every_source_is_packaged():
    """An installed copy builds its library from the sources that came with it."""
    meta = tomllib.loads((Path(__file__).resolve().parent.parent / "pyproject.toml").read_text())
    patterns = meta["tool"]["setuptools"]["package-data"]["cornstarch_b200.csrc"]
    for src in (*B.sources(), *B._headers(), B.HOST_OPS_SRC):
        assert any(fnmatch.fnmatch(src.name, p) for p in patterns), src.name
