"""A program that ends with renderers and results still alive ends quietly (its
functions keep its globals until the package's own are gone)."""
import os
import subprocess
import sys

import pytest

import helpers

PROGRAM = """
import sys
import torch
sys.path.insert(0, {tests!r})
import helpers
ve = helpers.package()
words, depth, mats, cam, fc = helpers.small_setup()
fc.width, fc.height = 300, 200


def images_of(r):
    r.set_materials(mats)
    sid = r.upload_scene(words, depth)
    return [r.render(sid, cam, fc) for _ in range(3)]


keep = [ve.Renderer(hash_log2=12) for _ in range(2)]
keep += [images_of(r) for r in keep]
print("rendered")
"""


@pytest.mark.gpu
def test_exit_with_renderers_alive():
    tests = os.path.join(helpers.ROOT, "tests")
    p = subprocess.run([sys.executable, "-c", PROGRAM.format(tests=tests)], capture_output=True, text=True, timeout=300)
    assert p.returncode == 0 and p.stdout.split() == ["rendered"]
    assert "Exception" not in p.stderr and "Traceback" not in p.stderr, p.stderr
