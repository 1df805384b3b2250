"""Rules of the CUDA sources that no run can show without a hang."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "cuteafd_b200" / "csrc"


@pytest.mark.parametrize("name,sections", [("attention_mla_prefill.cu", 3), ("attention_prefill_pair.cuh", 1)])
def test_warps_give_up_as_a_whole_in_front_of_warp_collectives(name, sections):
    """The softmax warps read and write tensor memory (`tcgen05.ld` / `st`, warp collectives) behind their waits, so a wait that ran out must end
    all lanes: they wait by vote (`mbar_wait_warp`), not lane by lane."""
    text = (CSRC / name).read_text()
    parts = re.findall(r"^struct PfRow .*?^\};|-- softmax \+ epilogue.*?__syncthreads\(\);", text, re.S | re.M)
    assert len(parts) == sections
    for part in parts:
        assert "mbar_wait_warp(" in part and "mbar_wait_bounded(" not in part
