"""When the host polls the error words after a step (csrc/error_words.h), compiled for the host with and without the phase traces."""
import os
import subprocess

import pytest
from conftest import ROOT

PROGRAM = r"""
#include "error_words.h"
#include <cstdio>
int main() {
  std::printf("%d%d%d%d", orion::poll_after_step(true, 0), orion::poll_after_step(true, 4), orion::poll_after_step(false, 0), orion::poll_after_step(false, 1));
}
"""


@pytest.mark.parametrize("flags,expected", [([], "0111"), (["-DORION_TRACE"], "1111")])
def test_steps_that_poll(tmp_path, flags, expected):
    """A step of a build with traces always polls: the polling functions are what switches the traces on and prints them."""
    source, program = tmp_path / "words.cpp", tmp_path / "words"
    source.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", *flags, "-I", os.path.join(ROOT, "orionserve-rs_b200", "csrc"), str(source), "-o", str(program)], check=True)
    assert subprocess.run([str(program)], stdout=subprocess.PIPE, text=True, check=True).stdout == expected
