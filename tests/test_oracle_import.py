"""Importing the oracle changes nothing for the process that does it: the benchmark times its matmuls."""

import os
import subprocess
import sys
from pathlib import Path


def test_import_leaves_the_environment_alone():
    env = {k: v for k, v in os.environ.items() if k != "MKL_CBWR"}
    code = "import os; import oracle.lane_oracle; assert dict(os.environ).get('MKL_CBWR') is None"
    subprocess.run([sys.executable, "-c", code], cwd=Path(__file__).resolve().parent.parent, env=env, check=True)
    assert os.environ["MKL_CBWR"] == "COMPATIBLE"            # what the comparisons with pinned outputs run under
