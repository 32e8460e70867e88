"""How a plain plan launches its sweeps, as a function of the mode it is created
for (host, no GPU).

A plan of several rounds per launch keeps two copies of A and a persistent one
rotates a single copy in place, so a plan must be one of them: the choice is
one value, made from arguments.  The process-wide mode can change between two
reads, and a plan built from two different values held both forms; so the
library reads it in one place only.
"""
import os
import re

import pytest

import jsvd
from conftest import PKG

SHAPES = [(1, 1), (2, 2), (5, 5), (64, 48), (256, 256), (257, 20), (512, 512), (1000, 333), (1024, 1024), (1025, 64),
          (4096, 1024)]


@pytest.mark.parametrize("m,n", SHAPES)
@pytest.mark.parametrize("threads", [32, 256, 1024])
def test_one_form_per_mode(m, n, threads):
    for coop in (False, True):
        for mode in range(4):
            form, rounds, slots = jsvd.plain_sweep_form(m, n, threads, mode, cooperative=coop)
            fused = mode == 0 and threads == 256 and n >= 5 and m <= 1024
            assert form == (1 if fused else 2 if mode == 1 and coop and n >= 2 else 0)
            assert (rounds > 0 and slots > 0) == (form == 1)


@pytest.mark.parametrize("n", [5, 6, 100, 640, 1024])
def test_fused_shape_fits_a_block(n):
    for m in (n, 1024):
        form, rounds, slots = jsvd.plain_sweep_form(m, n)
        assert form == 1
        threads = 32 if m <= 256 else 64
        assert threads * (slots + rounds - 1) <= 512
        assert rounds <= (n + 1) // 2 - 1
        assert slots * 148 >= (n + 1) // 2


def test_the_process_wide_mode_is_read_once_per_plan():
    """acquire_plain_plan reads it (and the ABI's getter); a plan's creation does not."""
    def mentions(name):
        text = re.sub(r"//[^\n]*", "", open(os.path.join(PKG, "csrc", name)).read())
        return len(re.findall(r"(?<!\w)sweep_mode\(\)", text))

    assert mentions("plain.cu") == 1  # its definition
    assert mentions("abi.cu") == 2


def test_argument_errors():
    for args in [(2, 3, 256, 0), (0, 0, 256, 0), (4, 3, 256, 4), (4, 3, 256, -1)]:
        with pytest.raises(jsvd.InvalidArgument):
            jsvd.plain_sweep_form(*args)
    with pytest.raises(jsvd.InvalidArgument):
        jsvd.plain_sweep_form(4, 3, sms=0)
