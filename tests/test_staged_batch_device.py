"""The kernel that stages a step's batch runs on the batch's device, whichever is current, and only where that is a GPU."""
import contextlib

import torch

from cme213_final_project_b200 import ops
from cme213_final_project_b200.graph import GraphedStep


class OnOtherDevice:
    """What the staging looks at of a contiguous int32 tensor on the second GPU."""
    device, dtype, shape, is_cuda = torch.device("cuda", 1), torch.int32, torch.Size([64]), True

    is_contiguous = lambda self: True                                        # noqa: E731
    numel = lambda self: 64                                                  # noqa: E731
    data_ptr = lambda self: 256                                              # noqa: E731


def test_launches_on_the_device_of_the_batch(monkeypatch):
    current, seen = [0], []

    @contextlib.contextmanager
    def device(d):
        before, current[0] = current[0], torch.device(d).index
        yield
        current[0] = before

    class Lib:
        @staticmethod
        def cme_copy_pair_i32(*args):
            seen.append((current[0], args[4], args[5]))
            return 0

    monkeypatch.setattr(torch.cuda, "device", device)
    monkeypatch.setattr(ops, "lib", lambda: Lib)
    monkeypatch.setattr(ops, "_st", lambda: 1000 + current[0])
    GraphedStep._stage(None, *(OnOtherDevice() for _ in range(4)))
    assert seen == [(1, 64, 1001)] and current == [0]


def test_batches_in_host_memory_are_copied_as_they_are():
    step = GraphedStep(lambda x, y: None, 8, 1, torch.device("cpu"))
    x, y = torch.arange(8, dtype=torch.int32), torch.arange(8, 16, dtype=torch.int32)
    step._stage(step.static_x[0], x, step.static_y[0], y)
    assert torch.equal(step.static_x[0], x) and torch.equal(step.static_y[0], y)
