"""What holds of the kernels' sources by reading them."""

from pathlib import Path

import pytest

SOURCES = Path(__file__).resolve().parents[1] / "miniserve-llm-nv_b200" / "csrc"


@pytest.mark.parametrize("name", ["attention_decode.cu", "attention_latent_decode.cu", "attention_latent_tcgen05.cu", "experts_tcgen05.cu"])
def test_a_kernel_that_gives_up_lets_its_copies_land(name):
    """Bulk copies into shared memory outlive the thread that asked for them: where a bounded wait gives up, the copies in flight are
    waited for (again with a bound) before the block exits."""
    text = (SOURCES / name).read_text()
    assert "mbar_expect_tx(" in text
    assert "let_copies_land(" in text
