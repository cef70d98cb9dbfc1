"""What the step kernels read before they wait for the kernel (or cluster phase) before them: nothing that a
step kernel writes. A kernel that starts early is promised the writes of the earlier ones only once it has
waited, so this is checked on the sources."""
import re
from pathlib import Path

import pytest

SOURCE = (Path(__file__).resolve().parents[1] / "arbo_gpu_fit_gb300" / "csrc" / "kernels.cu").read_text()

# Arrays of a simulation that its step kernels write.
WRITTEN = {"n_born", "n_dtime", "n_next", "n_status", "n_exposed", "n_recovery", "n_ple", "n_strain", "n_imm",
           "m_code", "m_stat", "m_life", "m_exposed", "m_strain", "ledger", "infh", "infm", "inc", "mcnt", "transh",
           "transm", "winh", "winm", "s_ninc", "s_ninf", "s_one", "s_ncount", "s_mcount", "s_minf", "s_spatial"}


def body(name):
    """The text of function `name`, from its opening to its closing brace."""
    m = re.search(r"\b" + name + r"\([^;{]*\)\s*\{", SOURCE)
    assert m, name
    depth = 0
    for i in range(m.end() - 1, len(SOURCE)):
        depth += {"{": 1, "}": -1}.get(SOURCE[i], 0)
        if depth == 0:
            return re.sub(r"//[^\n]*", "", SOURCE[m.end():i])
    raise AssertionError(name)


def members(text):
    return set(re.findall(r"\bd\.(\w+)", text))


@pytest.mark.parametrize("name", ["foi_series", "foi_events", "infect_unit", "demog_mosquito_quad"])
def test_reads_before_the_wait_are_of_constant_data(name):
    text = body(name)
    assert text.count("wait();") == 1, "one wait for all that follows"
    early = text.split("wait();")[0]
    assert not members(early) & WRITTEN


def test_start_of_a_quad_reads_constant_data():
    # demog_mosquito_quad calls it before its wait.
    assert not members(body("quad_start")) & WRITTEN


def test_list_of_written_arrays_is_complete():
    # Every array that a step body stores to, or gives to an atomic, is in the list above.
    stored = set()
    for name in ("human_due", "mosq_deep", "mosquito_quad_core", "split_events", "foi_series", "foi_events",
                 "infect_human", "infect_mosquito", "infect_unit"):
        text = body(name)
        stored |= set(re.findall(r"\bd\.(\w+)\[[^;=]*\]\s*=[^=]", text))
        stored |= set(re.findall(r"atomic\w+\(&d\.(\w+)\[", text))
        stored |= set(re.findall(r"counter_dec\(&d\.(\w+)\[", text))
    assert {"ledger", "mcnt", "infh", "n_status", "m_code", "transh", "winm"} <= stored
    assert stored <= WRITTEN
