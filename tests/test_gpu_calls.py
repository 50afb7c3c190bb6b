"""A call reads its inputs and writes its results where they are: whatever form an input comes in, the
same bits, in fresh tensors."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp32", "tf32", "bf16"])
@pytest.mark.parametrize("case", ["linear_1x3072x768", "layernorm_2048x768", "mlp_2048", "gpt2_block_t128", "block_d64"])
def test_every_form_of_input_gives_the_same_results(case, precision):
    from gpu_helpers import build_executable
    from helpers import case_data, load_plan

    plan = load_plan(case)
    (x,), consts, _ = case_data(case, plan)
    exe = build_executable(case, precision, plan_json=plan, consts=consts)
    x = torch.from_numpy(np.ascontiguousarray(x))
    exe.static_inputs[0].copy_(x)
    exe.run_static()
    want = exe.static_outputs[0].clone()
    dense = x.cuda()
    unaligned = torch.empty(x.numel() + 1, device="cuda")[1:].view(x.shape).copy_(x)
    strided = torch.empty(x.shape[::-1], device="cuda").t().copy_(x)
    held = []
    for form in (dense, x, unaligned, strided, x.double(), dense.clone(), dense):
        before = form.clone()
        held.append(exe(form)[0])
        assert torch.equal(form, before)
    exe.run_static()                       # the fixed buffers again, after calls on others
    held.append(exe.static_outputs[0])
    sink = torch.empty_like(want)
    exe.run_on([dense], [sink])
    in_place = dense.clone()
    if in_place.shape == want.shape:
        exe.run_on([in_place], [in_place])
        held.append(in_place)
    torch.cuda.synchronize()
    exe.status()
    for got in held + [sink]:
        assert torch.equal(got, want)
    assert len({t.data_ptr() for t in held}) == len(held)
    with pytest.raises(ValueError):
        exe(dense[:, :-1])
    with pytest.raises(TypeError):
        exe(dense, dense)


@pytest.mark.parametrize("case", ["linear_128x768x768", "linear_2048x3072x768"])
def test_calls_from_a_thread_that_has_used_no_gpu(case):
    """The first call of a thread may be one on buffers of its own; the next call finds the plan whole."""
    import threading

    from gpu_helpers import build_executable

    exe = build_executable(case, "tf32")
    x = torch.randn(exe.input_shapes[0], device="cuda")
    exe.static_inputs[0].copy_(x)
    exe.run_static()
    want = exe.static_outputs[0].clone()
    torch.cuda.synchronize()
    got = []
    thread = threading.Thread(target=lambda: got.extend(exe(x)))
    thread.start()
    thread.join()
    exe.static_outputs[0].zero_()
    exe.run_static()
    torch.cuda.synchronize()
    exe.status()
    assert torch.equal(exe.static_outputs[0], want)
    assert len(got) == 1 and torch.equal(got[0], want)


@pytest.mark.parametrize("case,precision", [("layernorm_2048x768", "fp32"), ("linear_128x768x768", "tf32"), ("linear_2048x3072x768", "bf16"),
                                            ("mlp_2048", "bf16")])
def test_calls_from_several_threads_keep_to_their_own_tensors(case, precision):
    """On one stream the calls of a module run one after the other, whichever thread they come from."""
    import threading

    from gpu_helpers import build_executable

    exe = build_executable(case, precision)
    inputs = [torch.randn(exe.input_shapes[0], device="cuda") for _ in range(6)]
    inputs[3:] = [x.t().contiguous().t() for x in inputs[3:]]      # (read through the fixed buffer)
    want = [exe(x)[0] for x in inputs]
    torch.cuda.synchronize()
    right = []

    def calls(x, y):
        right.append(sum(torch.equal(exe(x)[0], y) for _ in range(50)))

    threads = [threading.Thread(target=calls, args=pair) for pair in zip(inputs, want)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    exe.status()
    assert right == [50] * 6


def test_a_tensor_without_memory_is_read_as_its_values():
    """Zeros that have no memory to point at are copied; what an earlier call left in the fixed buffer is not used."""
    from gpu_helpers import build_executable

    exe = build_executable("layernorm_2048x768", "fp32")
    x = torch.randn(exe.input_shapes[0], device="cuda")
    want = exe(torch.zeros_like(x))[0]
    none = torch._efficientzerotensor(exe.input_shapes[0], device="cuda")
    exe(x.cpu())
    assert torch.equal(exe(none)[0], want)
    exe(x.cpu())
    sink = torch.empty_like(want)
    exe.run_on([none], [sink])
    assert torch.equal(sink, want)


def test_requests_bring_the_first_input_of_a_module_with_more():
    """A step's sources are first inputs and its sinks first outputs; the others are the module's fixed buffers."""
    from kiln_b200.codegen import program_from_plan
    from kiln_b200.runtime import GPUExecutable, StreamedBatch
    from kiln_b200.spec import KernelSpec, NodeSpec, OperandSpec, PlanSpec

    shape = (40, 64)

    def module():
        at = lambda base, i: OperandSpec((base, i), 0, shape, (64, 1))     # noqa: E731
        kernels = [KernelSpec(f"k{i}", "elementwise", [NodeSpec(op, [("operand", 0), ("operand", 1)], shape, {})], [at("input", 0), at("input", 1)],
                              [(0, at("output", i))]) for i, op in enumerate(["add", "sub"])]
        plan = PlanSpec("sum_and_difference", [shape, shape], [shape, shape], 0, {}, kernels)
        return GPUExecutable(program_from_plan(plan, "fp32"), 0, {}, plan.input_shapes, plan.output_shapes, cuda_graphs=False)

    modules = [module() for _ in range(2)]
    sources = [torch.randn(shape, device="cuda") for _ in range(4)]
    sinks = [torch.empty(shape, device="cuda") for _ in range(4)]
    for i, m in enumerate(modules):
        m.static_inputs[1].fill_(1.0 + i)
    StreamedBatch(modules).capture(sources, sinks).run()
    torch.cuda.synchronize()
    for i, (x, y) in enumerate(zip(sources, sinks)):
        assert torch.equal(y, x + (1.0 + i % 2))
    assert torch.equal(modules[1].static_outputs[1], sources[3] - 2.0)


def test_a_result_that_autograd_watches_is_refused():
    """Writing into a leaf that requires a gradient is an error, and so is a backward pass over a tensor written since."""
    from gpu_helpers import build_executable

    exe = build_executable("layernorm_2048x768", "fp32", cuda_graphs=False)
    x = torch.randn(exe.input_shapes[0], device="cuda")
    with pytest.raises(RuntimeError, match="requires grad"):
        exe.run_on([x], [torch.empty_like(x).requires_grad_()])
    saved = torch.empty_like(x)
    loss = (saved * torch.ones_like(x).requires_grad_()).sum()
    exe.run_on([x], [saved])
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        loss.backward()


@pytest.mark.parametrize("beyond", [0, 1])
def test_both_sides_of_the_limit_of_direct_calls(beyond):
    """A plan of as many launches as are enqueued directly, and one of one more, which replays a graph: the same results."""
    from kiln_b200 import runtime
    from kiln_b200.codegen import program_from_plan
    from perf import cases

    rows, d, n = 37, 260, runtime.DIRECT_LAUNCHES + beyond
    p = cases._Plan("norms", (rows, d), (rows, d))
    x = p.x
    for i in range(n):
        y = p.y if i + 1 == n else p.buffer(rows, d)
        p.layernorm(x, f"{i}.", y)
        x = y
    plan = p.spec()
    consts = cases._constants(plan.const_shapes, np.random.default_rng(0))
    exe = runtime.GPUExecutable(program_from_plan(plan, "fp32"), plan.arena_bytes, consts, plan.input_shapes, plan.output_shapes)
    assert exe.device_launches == n and (exe._caller is None) == bool(beyond)
    inputs = [torch.randn(rows, d, device="cuda") for _ in range(3)]
    outputs = [exe(x)[0] for x in inputs]
    for x, got in zip(inputs, outputs):
        exe.static_inputs[0].copy_(x)
        exe._launch()
        assert torch.equal(exe.static_outputs[0], got)
