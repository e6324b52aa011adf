"""What the source of kernels that may start early has to keep to, checked on the CPU.

A kernel launched with fb::launch_dependent runs while the kernel before it still writes. The
language lets a compiler move a load of memory that it takes for unchanging (a `const
__restrict__` kernel parameter, or __ldg) above fb::dependency_wait(); whether one does shows in
no test that happens to pass. So the source is held to the rule that makes such a load
impossible: these parameters are replaced by fb::after_wait() of themselves behind the wait.
"""

import re
from pathlib import Path

import pytest

SOURCES = sorted((Path(__file__).parent.parent / "flint_b200" / "csrc").glob("*.cu"))


def kernels(text):
    """(name, parameters, body) of every __global__ function."""
    text = re.sub(r"//[^\n]*", "", text)
    for head in re.finditer(r"__global__", text):
        opening = re.compile(r"(\w+)\s*\(").search
        at = head.end()
        while True:
            found = opening(text, at)
            depth, end = 1, found.end()
            while depth:
                depth += {"(": 1, ")": -1}.get(text[end], 0)
                end += 1
            if found.group(1) in ("__launch_bounds__", "__cluster_dims__"):
                at = end
                continue
            break
        parameters = text[found.end():end - 1]
        begin = text.index("{", end)
        depth, stop = 1, begin + 1
        while depth:
            depth += {"{": 1, "}": -1}.get(text[stop], 0)
            stop += 1
        yield found.group(1), parameters, text[begin:stop]


def waiting_kernels():
    for path in SOURCES:
        for name, parameters, body in kernels(path.read_text()):
            if "dependency_wait()" in body:
                yield pytest.param(parameters, body, id=f"{path.stem}:{name}")


def test_the_scan_finds_the_kernels():
    names = {p.id.split(":")[1] for p in waiting_kernels()}
    assert {"fb_layernorm_forward_regs", "fb_softmax_cross_entropy_rolling", "fb_column_partials",
            "fb_layernorm_backward_dx", "fb_gemm_tn_reduce", "fb_column_finish", "fb_heads_move",
            "fb_decode_linear", "fb_attention_forward", "fb_embedding_prepare"} <= names


@pytest.mark.parametrize("parameters, body", list(waiting_kernels()))
def test_inputs_are_read_behind_the_wait(parameters, body):
    behind = body[body.index("dependency_wait()"):]
    for parameter in parameters.split(","):
        declared = re.search(r"\bconst\b.*\*\s*__restrict__\s+(\w+)\s*$", parameter.strip(), re.S)
        if declared:
            name = declared.group(1)
            assert re.search(rf"\b{name} = fb::after_wait\({name}\);", behind), name


@pytest.mark.parametrize("path", SOURCES, ids=lambda p: p.stem)
def test_no_loads_that_ask_for_unchanging_memory(path):
    text = re.sub(r"//[^\n]*", "", path.read_text())
    assert "__ldg(" not in text


@pytest.mark.parametrize("parameters, body", list(waiting_kernels()))
def test_a_kernel_releases_the_next_one_behind_its_own_wait(parameters, body):
    # So that whatever a kernel depends on is over before the one after the next can begin.
    assert "dependency_release()" in body
    assert body.index("dependency_wait()") < body.index("dependency_release()")


def test_kernels_that_read_before_their_wait_stand_behind_an_ordinary_launch():
    """The decode kernels read weights, the position and older cache rows ahead of their wait: the
    chain that they end has to begin with a launch that waits for everything before it."""
    text = (SOURCES[0].parent / "generate.cu").read_text()
    for function, first, then in (("enqueue_step", "fb_decode_embed", "run_token("),
                                  ("flint_b200_generator_prefill", "fb_take_last_rows", "run_head(")):
        body = text[re.search(rf"flint_status {function}\(", text).start():]
        body = body[:body.index("\n}\n")]
        assert f"{first}<<<" in body and body.index(f"{first}<<<") < body.index(then)
        between = body[body.index(f"{first}<<<"):body.index(then)]
        assert "launch_dependent" not in between


def function_body(text, name):
    body = text[re.search(rf"\n\S[^\n;]*\b{name}\(", text).start():]
    return body[:body.index("\n}\n")]


def launches_in_order(body):
    """The launching calls of a function of generate.cu, in source order."""
    return re.findall(r"\b(dense_weights|layernorm|decode_linear|linear<Act::\w+>|fb_cache_store|attention_forward|"
                      r"fb_decode_attention|flint_embedding_forward|run_prompt)\(", body.replace("fb_cache_store,", "fb_cache_store("))


def steady_weights_have_a_kernel_between(text):
    """linear() tells its GEMM that the weights are steady, so that it fetches some before its wait. What may have
    written them just before is dense_weights' expansion, or, ahead of a prompt, anything."""
    prompt = launches_in_order(function_body(text, "run_prompt"))
    expansion = prompt.index("dense_weights")
    first_gemm = next(i for i, name in enumerate(prompt) if name.startswith("linear<"))
    prefill = launches_in_order(function_body(text, "flint_b200_generator_prefill"))
    return (prompt.count("dense_weights") == 1 and first_gemm - expansion >= 2
            and prefill.index("flint_embedding_forward") < prefill.index("run_prompt"))


def test_weights_fetched_before_the_wait_were_written_a_kernel_earlier():
    text = re.sub(r"//[^\n]*", "", (SOURCES[0].parent / "generate.cu").read_text())
    assert steady_weights_have_a_kernel_between(text)
    # Only linear() says so, and it is called behind an expansion (above) or an ordinary launch
    # (test_kernels_that_read_before_their_wait_stand_behind_an_ordinary_launch).
    assert text.count("stream, true));") == 3 == function_body(text, "linear").count("stream, true));")
    gemm = re.sub(r"//[^\n]*", "", (SOURCES[0].parent / "gemm.cu").read_text())
    once = gemm[gemm.index("fb_gemm_once(const"):]
    ahead = once[:once.index("dependency_wait()")]
    assert re.findall(r"\bearly = ([^;]*);", ahead) == ["once.steady_b != 0 ? min(stages, blocks) : 0"]
    assert re.findall(r"&p\.map_\w", ahead.split("auto fetch_b")[1].split("};")[1]) == []


def test_the_check_notices_an_expansion_right_before_its_gemm():
    text = (SOURCES[0].parent / "generate.cu").read_text()
    expansion = re.search(r"\n *FB_TRY\(dense_weights\([^\n]*", text).group(0)
    norm = re.search(r"\n *FB_TRY\(layernorm\(g, l\.ln1_w[^\n]*", text).group(0)
    assert expansion + norm in text
    assert not steady_weights_have_a_kernel_between(text.replace(expansion + norm, norm + expansion))
