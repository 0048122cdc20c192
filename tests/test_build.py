"""A checkout without the shared object builds and loads in one call, with and without a GPU in the machine."""
import os
import shutil
import subprocess
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent


@pytest.mark.parametrize('gpu', [False, True])
@pytest.mark.parametrize('imported_before', [False, True])
def test_build_from_a_checkout_without_the_extension(tmp_path, gpu, imported_before):
    if not list((ROOT / 'build' / 'deepep_b200').glob('*.o')):
        pytest.skip('no object cache: the build would take a minute')
    if gpu and imported_before:
        pytest.skip('importing the package without the extension is an error on a machine with a GPU')
    ignore = shutil.ignore_patterns('*.so', '__pycache__')
    shutil.copytree(ROOT / 'deepep_b200', tmp_path / 'deepep_b200', ignore=ignore)
    shutil.copytree(ROOT / 'build', tmp_path / 'build', ignore=shutil.ignore_patterns('link.stamp'))     # (compiled objects; linking is done anew)
    shutil.copy(ROOT / '__graft_entry__.py', tmp_path)
    code = f'import torch\ntorch.cuda.is_available = lambda: {gpu}\n'
    if imported_before:
        code += 'import deepep_b200\nassert deepep_b200._C is None\n'
    code += 'import __graft_entry__ as entry\nentry.build()\nimport deepep_b200\nprint(deepep_b200._C.__file__)\n'
    env = dict(os.environ, PYTHONPATH=str(tmp_path))
    done = subprocess.run([sys.executable, '-c', code], cwd=tmp_path, env=env, capture_output=True, text=True, timeout=600)
    assert done.returncode == 0, done.stderr[-2000:]
    assert Path(done.stdout.split()[-1]).parent == tmp_path / 'deepep_b200'
