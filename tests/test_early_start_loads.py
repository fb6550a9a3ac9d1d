"""The forward pass starts beside the kernel that writes its quad image, so its
loads of that image are ordinary ones: the read-only path (__ldg, or a const
__restrict__ parameter, which the compiler takes for it) holds only for data that
nothing writes while the kernel runs.  Checked on the source."""
import os
import re

from imgrecsrc_b200 import build


def test_the_quad_image_is_not_read_through_the_read_only_path():
    text = open(os.path.join(build.CSRC, "projector.cu")).read()
    march = text[text.index("__device__ __forceinline__ void march_rows("):text.index("// The rows that the rays of a warp can meet")]
    assert "__ldg(" not in march and "__restrict__" not in march
    assert len(re.findall(r"load_quad<NC>\(", march)) == 10
    # only the persistent launches, which start after the image is complete, ask for that path
    assert "march_rows<FAN, MODE, R == kAllParts>(" in text
    for kernel in ("k_forward(", "double forward_rays("):
        sig = text[text.index(kernel):]
        assert "const float4 *quad" in sig[:sig.index("{")]
