"""Index ranges of the tensor sweeps' inboxes (gcs_mi_tensor.cu), from the
constants in the source: every longitude that a lane sends to, takes or reads,
in the steps that fill up the last group too, lies inside its own inbox."""
import os
import re

SOURCE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                      "gamera_cube_b200", "csrc", "gcs_mi_tensor.cu")


def test_inbox_ranges():
    text = open(SOURCE).read()
    pad = int(re.search(r"constexpr int kInboxPad = (\d+);", text).group(1))
    group = int(re.search(r"constexpr int kGroup = (\d+);", text).group(1))
    most = int(re.search(r"constexpr int kMaxLongitudes = (\d+);", text).group(1))
    body = re.search(r"constexpr int inbox_len\(int np\) \{ return (.*); \}", text).group(1)
    for np in range(2, most + 1):
        length = eval(body, {"np": np, "kInboxPad": pad, "kGroup": group})
        steps = -(-(np + 31) // group) * group
        forward = (0, steps - 1)                       # columns of a sweep
        reverse = (np + 30 - (steps - 1), np + 30)
        touched = {
            "sent forward by lane 31": (forward[0] - 31, forward[1] - 31),
            "sent in reverse by lane 0": reverse,
            "taken forward": forward,
            "taken in reverse": (reverse[0] - 31, reverse[1] - 31),
            "pole edges": reverse,
        }
        for what, (low, high) in touched.items():
            assert 0 <= low + pad and high + pad < length, (np, what, low, high)
