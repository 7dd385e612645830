"""The bookkeeping of csrc/decode_rows.cu on the CPU: what its source promises about barriers."""
import pathlib
import re

SOURCE = (pathlib.Path(__file__).resolve().parents[1] / "nano-qwen3tts-vllm_b200" / "csrc" / "decode_rows.cu").read_text()
CODE = re.sub(r"//[^\n]*", "", SOURCE)


def test_warps_meet_between_polling_and_the_next_barrier():
    """Lanes of a warp leave a polling loop one by one; an aligned barrier, a vote or a shuffle behind it wants all of them."""
    marks = [(m.start(), m.group(1)) for m in re.finditer(r"(dr_wait(?:_all)?(?=[(<])|dr_sync\(\)|__syncwarp\(\)|__syncthreads\(\)|__all_sync\(|warp_sum\()", CODE)]
    waits, open_wait = 0, None
    for at, name in marks:
        line = CODE[:at].count("\n") + 1
        if name.startswith("dr_wait"):
            if re.search(r"__forceinline__ \w+ $", CODE[:at]):
                continue                                         # its definition
            waits, open_wait = waits + 1, line
        elif name == "__syncwarp()":
            open_wait = None
        else:
            assert open_wait is None, f"{name} in line {line} follows the polling of line {open_wait}"
    assert waits >= 6
