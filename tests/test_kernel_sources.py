"""Rules of the CUDA sources that a run on a GPU shows only when something else has already gone wrong."""

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "rapid_llm_b200" / "csrc"


@pytest.mark.parametrize("name", ["moe_tc.cu", "attention_plane_tc.cuh"])
def test_copies_in_flight_are_waited_for_after_the_others_gave_up(name):
    """A wait under the block's abort flag gives up at once when the flag is set: the last wait for the copies has a flag of
    its own, and nothing skips it."""
    source = (CSRC / name).read_text()
    drain = source.index("volatile int go_on = 0;")
    loop = source[drain : source.index("\n    }\n", drain)]
    waits = re.findall(r"mbar_wait\((.*)\);", loop)
    assert waits and all("&go_on" in wait and "aborted" not in wait for wait in waits)
    assert "*aborted" not in source[source.rindex("tma_load_2d(", 0, drain) : drain]


# what no kernel of a step writes: weights, tables made when the weights are loaded, the step's uploaded metadata
STEADY = {"w", "wq", "wc", "bias", "correction", "weight", "ln_weight", "ln_bias", "taps", "rate", "mu", "pq", "freq", "inv_freq",
          "cu_seqlens", "entry_slot", "entry_start", "positions", "kv_dest"}


@pytest.mark.parametrize("name", ["moe.cu", "moe_tc.cu", "latent.cu", "recurrent.cu"])
def test_what_a_step_writes_is_not_read_as_invariant(name):
    """A load through a const restrict pointer may be moved above the wait for the kernel before."""
    invariant = set(re.findall(r"const [\w:]+\* ?__restrict__ (\w+)", (CSRC / name).read_text()))
    assert invariant <= STEADY, sorted(invariant - STEADY)


def test_a_permission_is_remembered_per_device():
    """A kernel's shared memory beyond 48 KB belongs to the current device: what remembers that it was asked for has a bit for
    each (`allow_shared`), and nothing a flag for the process."""
    for path in sorted(CSRC.glob("*.cu*")):
        assert not re.search(r"\bbool\b[^;\n]*configured", path.read_text()), path.name
