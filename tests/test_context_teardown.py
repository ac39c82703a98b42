"""A call that failed may leave an upload on the side stream, into the workspace and
from the pinned tables: both streams are waited for before either is given back."""
from pathlib import Path

API = Path(__file__).resolve().parent.parent / "entropical_gb300" / "csrc" / "api.cu"


def body(signature):
    text = API.read_text()
    a = text.index(signature + " {")
    return text[a:text.index("\n}\n", a)]


def test_begin_call_waits_for_both_streams_before_it_resets_the_workspace():
    b = body("int Ctx::begin_call()")
    reset = b.index("arena.reset()")
    assert b.index("cudaStreamSynchronize(stream)") < reset
    assert b.index("cudaStreamSynchronize(side_stream)") < reset


def test_destroy_waits_for_both_streams_before_it_frees():
    b = body("void ent_destroy(ent_ctx* ctx)")
    first = min(b.index(f) for f in ("arena.release()", "cudaFree(", "cudaFreeHost(",
                                     "cudaStreamDestroy("))
    assert b.index("cudaStreamSynchronize(c->stream)") < first
    assert b.index("cudaStreamSynchronize(c->side_stream)") < first
