"""make_ref.py --if-present: sources that are all absent are passed over, a
checkout that has lost one of its files is an error."""
import os
import subprocess
import sys

import pytest

from conftest import ORACLE


@pytest.mark.parametrize("files,ok", [((), True), (("3dmhdsub.f",), False), (("3dmhdparam.f",), False)])
def test_if_present(tmp_path, files, ok):
    for f in files:
        (tmp_path / f).write_text("      END\n")
    r = subprocess.run([sys.executable, os.path.join(ORACLE, "make_ref.py"), "--if-present", "--src", str(tmp_path),
                        "--out", str(tmp_path / "out")], capture_output=True, text=True)
    assert (r.returncode == 0) == ok, r.stderr
