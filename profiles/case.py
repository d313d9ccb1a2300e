"""Three passes of a workload of perf/cases.py, steps stage by stage: what the ncu
commands of these summaries run.

    python profiles/case.py NAME [KEY=VALUE ...]     (e.g. learned_16m n=4194304)
"""
import os
import sys

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
from perf.cases import listed, prepare, run  # noqa: E402


def main():
    case = next(c for c in listed() if c["name"] == sys.argv[1])
    for pair in sys.argv[2:]:
        key, value = pair.split("=")
        case[key] = type(case[key])(value)
    state = prepare(case, 1)
    for _ in range(3):
        if state["kind"] == "step":
            print(state["sim"].step_profiled(state["params"]))
        else:
            run(state)


if __name__ == "__main__":
    main()
