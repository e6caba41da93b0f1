"""Memory that only makes steps faster is asked for after what a case needs."""
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "flowlb_b200" / "csrc"


def test_streams_form_creates_its_handles_before_their_second_buffers():
    text = (CSRC / "batch.cu").read_text()
    body = text[text.index("flb_status streams_setup("):text.index("flb_status case_state_copy(")]
    assert body.index("create_handle(") < body.index("b->d_second")
