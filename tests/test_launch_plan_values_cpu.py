"""Values that change between steps reach the calls of a recorded segment."""
from terapipe_b200.runtime.launch_plan import RecordingLibrary, SegmentCache


class _Lib:
    def __init__(self):
        self.calls = []

    def tp_update(self, lr):
        self.calls.append(("update", lr))
        return 0

    def tp_forward(self):
        self.calls.append(("forward",))
        return 0


def test_a_segment_is_recorded_again_when_its_values_change():
    real = _Lib()
    lib = RecordingLibrary(real)
    plan = SegmentCache(lib)
    derived = []

    def forward():
        derived.append("forward")
        lib.tp_forward()

    def update(lr):
        derived.append("update")
        lib.tp_update(lr)

    for lr in (1.0, 1.0, 2.0, 2.0, 1.0):
        plan.run("forward", forward)
        plan.expect("update", (lr,))
        plan.run("update", update, lr)
    assert [c[1] for c in real.calls if c[0] == "update"] == [1.0, 1.0, 2.0, 2.0, 1.0]
    assert derived == ["forward", "update", "update", "update"]      # the other segment stays recorded
    assert plan.replayed == 4 + 2 and len(plan.segments) == 2
