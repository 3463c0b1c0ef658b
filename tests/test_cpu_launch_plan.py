"""What the batched entry points launch, without a GPU: csrc/host/fg_cuda_api.c over a CUDA layer that only
writes its launches down (tests/native/recorded_launches.c)."""
import ctypes
import shutil
import subprocess
from ctypes import POINTER, byref, c_char_p, c_uint32, c_void_p
from pathlib import Path

import pytest

from flash_gordon_b200 import FG_OK, LIBRARY_PATH, FgError, SampleArgs, SamplerConfig

ROOT = Path(__file__).resolve().parent.parent
CSRC = ROOT / "flash_gordon_b200" / "csrc"
SOMEWHERE = 1 << 20  # a 16-byte aligned address that nothing here looks at

TOP_K = SamplerConfig.make(temperature=0.8, top_p=0.9, top_k=20)
LOWERING = SamplerConfig.make(temperature=0.8, top_p=0.9, top_k=20, presence=0.5)
GREEDY = SamplerConfig.make(0.0, 1.0, 1)


@pytest.fixture(scope="module")
def plan(library, tmp_path_factory):
    """plan(configs, rows, ...) -> (status, launches): one call, its launches as lines."""
    if shutil.which("gcc") is None:
        pytest.skip("no C compiler")
    path = tmp_path_factory.mktemp("plan") / "libplan.so"
    build = subprocess.run(
        ["gcc", "-std=c17", "-D_GNU_SOURCE", "-O1", "-shared", "-fPIC", "-Wl,-Bsymbolic", "-I", str(ROOT / "include"),
         "-I", str(CSRC / "cuda"), "-I", str(CSRC / "host"), str(CSRC / "host" / "fg_cuda_api.c"),
         str(ROOT / "tests" / "native" / "recorded_launches.c"), str(LIBRARY_PATH), f"-Wl,-rpath,{LIBRARY_PATH.parent}",
         "-lm", "-o", str(path)], capture_output=True, text=True)
    assert build.returncode == 0, build.stderr
    lib = ctypes.CDLL(str(path))
    lib.recorded_launches.restype = c_char_p
    err = FgError()
    context = c_void_p()
    assert lib.fg_cuda_context_create(0, byref(context), byref(err)) == FG_OK

    def call(configs, rows, vocab=151_936, dtype="f32", history=0, offset=0, uniforms=SOMEWHERE, shard=0, flags=1):
        array = (SamplerConfig * len(configs))(*configs)
        a = SampleArgs(logits=SOMEWHERE + offset * (4 if dtype == "f32" else 2), dtype=0 if dtype == "f32" else 1, rows=rows,
                       vocab=vocab, flags=flags, row_stride=vocab, config_count=len(configs), uniforms=uniforms,
                       configs=ctypes.cast(array, POINTER(SamplerConfig)), tokens=SOMEWHERE, token_logits=SOMEWHERE,
                       row_status=SOMEWHERE, history_max=history)
        if history:
            a.history_tokens = a.history_offsets = SOMEWHERE
        lib.recorded_clear()
        if shard:
            status = lib.fg_cuda_shard_topk(context, byref(a), c_uint32(0), c_uint32(vocab), c_uint32(shard), c_void_p(SOMEWHERE),
                                            c_void_p(SOMEWHERE), byref(err))
        else:
            status = lib.fg_cuda_sample_batch(context, byref(a), byref(err))
        return status, lib.recorded_launches().decode().splitlines()

    call.context, call.lib = context, lib
    yield call
    lib.fg_cuda_context_destroy(context)


def test_draws_that_no_row_uses_are_not_read(plan):
    """Greedy rows and the shard step take no draws; a caller may leave anything in `uniforms`."""
    for rows, vocab in ((1, 151_936), (64, 151_936), (1024, 151_936), (3, 2_000_000)):
        for offset in (0, 1):
            for configs, shard in (([GREEDY], 0), ([TOP_K], 20), ([LOWERING], 20), ([GREEDY], 1)):
                status, launches = plan(configs, rows, vocab, offset=offset, shard=shard, history=64)
                assert status == FG_OK and launches and all(l.endswith("uniforms=0") for l in launches), launches
            status, launches = plan([TOP_K], rows, vocab, offset=offset)
            assert status == FG_OK and all(l.endswith("uniforms=1") for l in launches), launches


def kernels(launches):
    return [line.split()[0] for line in launches]


@pytest.mark.parametrize("rows,vocab,dtype,offset,kernel", [
    (1, 151_936, "f32", 0, "team"), (296, 151_936, "f32", 0, "team"), (320, 151_936, "f32", 0, "ring"),
    (444, 151_936, "f32", 1, "ring"), (512, 151_936, "f32", 0, "team"), (512, 151_936, "f32", 1, "team"),
    (640, 128_256, "f32", 0, "ring"), (592, 128_256, "f32", 0, "team"), (400, 100_000, "f32", 0, "team"),
    (400, 151_936, "bf16", 0, "team"), (1024, 151_936, "f32", 0, "ring"), (1024, 151_936, "f32", 1, "team"),
    (1024, 151_936, "bf16", 0, "team"), (800, 100_352, "f32", 0, "team"), (2, 1_048_576, "f32", 0, "team"),
])
def test_kernel_of_a_lowering_batch(plan, rows, vocab, dtype, offset, kernel):
    """Long fp32 rows whose last wave of teams would be half empty, and large aligned fp32 batches, are the ring kernel's."""
    for configs, history in (([TOP_K], 0), ([LOWERING], 512)):
        status, launches = plan(configs, rows, vocab, dtype, history, offset)
        assert status == FG_OK and kernels(launches) == [kernel], launches


def mixed(rows, every, odd=None):
    """One row in `every` raises; `odd` overrides the last of those."""
    configs = [SamplerConfig.make(temperature=0.8, top_p=0.9, top_k=20, presence=-0.4 if r % every == 0 else 0.4) for r in range(rows)]
    if odd:
        configs[(rows - 1) // every * every] = SamplerConfig.make(temperature=0.8, top_p=0.9, top_k=20, **odd)
    return configs


@pytest.mark.parametrize("offset", [0, 1])
def test_kernels_of_a_batch_with_some_raising_rows(plan, offset):
    rows, vocab = 400, 151_936
    status, launches = plan(mixed(rows, 8), rows, vocab, history=512, offset=offset)
    assert status == FG_OK and [line.split()[:2] for line in launches] == [["team", "which=1"], ["team", "which=2"]]
    # a charge that does not grow with the count, an extreme factor, a history over half the vocabulary
    for odd, history in ((dict(frequency=-0.5), 512), (dict(repetition=2.0 ** -41), 512), (dict(repetition=2.0 ** 41), 512),
                         (None, vocab // 2 + 1)):
        status, launches = plan(mixed(rows, 8, odd), rows, vocab, history=history, offset=offset)
        assert status == FG_OK
        assert [line.split()[:2] for line in launches] == [["ring", "skip_raising=1"], ["stream", "only_raising=1"]]
    # many raising rows, and a small batch: one launch
    assert kernels(plan(mixed(rows, 2), rows, vocab, history=512, offset=offset)[1]) == ["team"]
    assert kernels(plan(mixed(30, 8), 30, vocab, history=512, offset=offset)[1]) == ["team"]
    assert kernels(plan(mixed(30, 8, dict(frequency=-0.5)), 30, vocab, history=512, offset=offset)[1]) == ["stream"]


@pytest.mark.parametrize("team,chunk,form", [(0, 1024, 0), (3, 1024, 0), (16, 1024, 0), (2, 384, 0), (4, 200, 0), (1, 1024, 2)])
def test_plans_that_cannot_be_launched_are_refused(library, team, chunk, form):
    """Before anything is enqueued: no CTAs, a number that is no cluster's, columns that do not cover the row."""
    launch = (c_uint32 * 512)()  # (larger than fgk_stream_launch)
    launch[3], launch[4] = 1, 1000  # rows, vocab
    refused = library.fgk_launch_team_select(launch, c_uint32(team), c_uint32(chunk), c_uint32(form), c_uint32(0), None)
    assert refused == 1  # cudaErrorInvalidValue
