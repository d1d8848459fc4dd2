torch 2.11.0+cu128, cpython-312-x86_64-linux-gnu, cxx11 abi 1
-O2 -std=c++17 -fPIC -shared -ltorch_python -ltorch_cuda -ltorch_cpu -ltorch -lc10_cuda -lc10 -lflagattn_b200 -Wl,-rpath,$ORIGIN