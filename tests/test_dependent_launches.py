"""Programmatic dependent launches start before the launch that writes their
inputs has ended. Their kernels may take the read-only path (`__ldg`) only for
data that no launch writes: this reads the sources and finds every such load."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "the-powder-toy-rust-wgpu_b200", "csrc")

# Per file with code of dependent kernels: what they may read that way. A plan's
# constants (spectra, twiddles, the spectrum build's tables), the element
# tables, and the pixel map, which only launches read that may still run.
READ_ONLY = {
    "air.cu": {"pmap", "props"},
    "air.cuh": set(),
    "air_strip.cuh": set(),
    "grav_fft.cu": {"kern", "tw"},
    "grav_fft_mixed.cuh": {"t"},
    "grav_particles.cu": {"rec"},
}


@pytest.mark.parametrize("name", sorted(READ_ONLY))
def test_read_only_loads_are_of_constants(name):
    with open(os.path.join(CSRC, name)) as f:
        src = re.sub(r"//[^\n]*", "", f.read())
    used = {re.match(r"\(*([A-Za-z_]\w*(?:\.\w+)?)", a).group(1) for a in re.findall(r"__ldg\(([^;]*)", src)}
    assert used <= READ_ONLY[name], f"{name}: __ldg of {sorted(used - READ_ONLY[name])}"


def test_the_pixel_map_is_read_after_the_wait():
    """A canvas in NoUpdate mode without heat runs the settle pass alone, as a
    dependent of the launch that may have written the pixel map."""
    with open(os.path.join(CSRC, "air.cu")) as f:
        src = re.sub(r"//[^\n]*", "", f.read())
    assert "load_after_wait(pmap" in src and not re.search(r"__ldg\(\s*pmap", src)
