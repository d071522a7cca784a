"""Values made once per device (csrc/per_device.h), compiled for the host:
another device has its own, and threads that come at once get the finished
value of the one that made it."""
import subprocess
import textwrap
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent


def test_made_once_per_device_and_never_seen_half_made(tmp_path):
    src, exe = tmp_path / "pd.cpp", tmp_path / "pd"
    src.write_text(textwrap.dedent("""
        #include <atomic>
        #include <chrono>
        #include <cstdio>
        #include <thread>
        #include <vector>
        #include "per_device.h"
        struct Props { int sms = 0, smem = 0; };
        int main()
        {
            vvpt::PerDevice<Props> props;
            std::atomic<int> made{0}, wrong{0};
            std::vector<std::thread> th;
            for (int t = 0; t < 16; t++)
                th.emplace_back([&, t] {
                    const int dev = t % 3;
                    for (int k = 0; k < 1000; k++) {
                        const Props &p = props.get(dev, [&] {
                            Props q;
                            q.sms = 100 + dev;
                            std::this_thread::sleep_for(std::chrono::milliseconds(20));
                            q.smem = 1000 + dev;
                            made++;
                            return q;
                        });
                        wrong += p.sms != 100 + dev || p.smem != 1000 + dev;
                    }
                });
            for (auto &t : th)
                t.join();
            std::printf("%d %d\\n", made.load(), wrong.load());
        }"""))
    subprocess.run(["g++", "-O1", "-std=c++17", "-pthread", "-I", str(ROOT / "vviewer_gb300" / "csrc"), str(src), "-o",
                    str(exe)], check=True)
    assert subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout.split() == ["3", "0"]


def test_kernel_launches_keep_no_state_of_one_device():
    """No launch code keeps a kernel's attributes or a device's properties in a
    variable of the process."""
    for src in (ROOT / "vviewer_gb300" / "csrc").glob("*.cu"):
        for line in src.read_text().splitlines():
            if line.strip().startswith(("static int ", "static bool ", "static size_t ")):
                assert "(" in line, f"{src.name}: {line.strip()}"
