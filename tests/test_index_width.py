"""Work counts over packed rows pass 2^31 (46 heads of 128: from 5.8 M rows on, which the entry points accept and which needs
more memory than a test should take): read from the sources that they are formed in 64 bits."""

import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "decentrik_prime_b200", "csrc")


def test_attention_counts_rows_in_64_bits():
    text = open(os.path.join(CSRC, "nf4ll_attn.cu")).read()
    rope = text[text.index("rope_kernel("):text.index("attn_fwd_kernel(")]
    delta = text[text.index("attn_delta_kernel("):text.index("store_unrotated(")]
    launch = text[text.index("static int attn_forward_hd("):text.index("static int attn_backward_hd(")]
    for name, part in (("rope_kernel", rope), ("attn_delta_kernel", delta)):
        assert not re.search(r"\bint idx\b", part), name
        assert "static_cast<int64_t>(blockIdx.x) * 256" in part, name
    assert re.search(r"const int64_t work = static_cast<int64_t>\(", rope) and re.search(r"const int64_t work = static_cast<int64_t>\(", launch)
