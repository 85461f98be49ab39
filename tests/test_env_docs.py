"""Every environment variable in the integration guide's table is read by the library, and every one the library reads is
in the table."""

import glob
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_documented_variables_are_the_ones_read():
    with open(os.path.join(ROOT, "INTEGRATION.md")) as f:
        table = f.read().split("## 5. Environment variables", 1)[1]
    documented = set()
    for row in re.findall(r"^\|([^|]*)\|", table, re.M):
        documented.update(re.findall(r"`(CRDFFT_[A-Z0-9_]+)", row))
    read = set()
    for path in glob.glob(os.path.join(ROOT, "crd_b200", "csrc", "*")):
        if os.path.isfile(path):
            with open(path) as f:
                read.update(re.findall(r"(?:getenv|env_bytes|env_top_k)\(\"(CRDFFT_[A-Z0-9_]+)\"", f.read()))
    assert documented == read
